// The persistent frame kernel: one launch runs all the passes of a step.
//
// Its CTAs stay resident for the whole step and alternate between the tet
// phase of a pass (the chunk kernels' arithmetic, chunk_tets.cuh) and its
// node phase (node_update.cuh).  They need no barrier: every word that one
// CTA hands to another is 16 bytes, three floats and the tag of the pass it
// belongs to, stored and loaded as one relaxed 128-bit access, and a reader
// polls the words it needs until their tags are the pass's.
//   node -> tets   the state words (hi, lo) of a node, written by the CTA that
//                  owns it, read by the chunks that touch it;
//   tets -> node   a chunk's partial force (and Jacobi-diagonal) sum of a
//                  node, read by the node's owner;
//   CTA -> all     a CTA's share of |g|^2 (every pass) and of the energy
//                  (line-search passes).
// A word is overwritten only after its readers are known to be done: a node's
// next state follows the partials of every chunk that read the last one, a
// chunk's next partial follows the state formed from the last one, and the
// |g|^2 words, which every CTA reads a pass later, alternate between two
// buffers.  Every CTA takes the line-search and pass decisions itself, from
// the same words in the same order, on its own shared-memory copy of the
// control block: the copies stay equal, and no kernel launch, host poll or
// "last CTA" tail sits between the passes.  The pass decision is deferred into
// the next pass, whose tets run on its foreseen outcome, and taken by a
// control warp beside the workers, so its sums leave the critical path.
//
// The arithmetic of a tet, a chunk's slot sums and a node's update is that of
// the pass kernels, and in the resident layout the order of every sum too
// (phybs_internal.cuh): positions, decisions and stats are theirs bit for bit.
// Walking CTAs add the energies of several chunks, so the walking layout's
// energy and |g|^2 agree with them to rounding (and are bit-reproducible).
//
// Two layouts (RES):
//   resident  every chunk has its own CTA, all of them co-resident; the
//             chunk's per-tet rows, corner records, local-node records and
//             (with incremental stress) base displacements are copied to
//             shared memory once a step, so a pass moves only the node words
//             and partials that change.  Any number of instances: each has
//             its own words and stops on its own.
//   walking   one instance of any size: CTA b walks the chunks b, b + G, ...
//             and reads their rows from global memory each pass.
//
// What bounds a pass: two exchanges through L2 and one tet's dependent chain;
// neither bandwidth nor issue.
#include <algorithm>

#include "../../include/phybs.h"
#include "chunk_tets.cuh"
#include "exchange.cuh"
#include "node_update.cuh"
#include "pass_ctl.cuh"
#include "pass_math.cuh"
#include "phybs_internal.cuh"

namespace pbs {

// A CTA's |g|^2 share: {value, tag}, one 64-bit access.
__device__ __forceinline__ uint2 ld_pair(const uint2 *p) {
    uint2 v;
    asm volatile("{\n\t.reg .b64 a;\n\tld.relaxed.gpu.global.b64 a, [%2];\n\tmov.b64 {%0, %1}, a;\n\t}"
                 : "=r"(v.x), "=r"(v.y)
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ void st_pair(uint2 *p, unsigned x, unsigned tag) {
    asm volatile("{\n\t.reg .b64 a;\n\tmov.b64 a, {%1, %2};\n\tst.relaxed.gpu.global.b64 [%0], a;\n\t}" ::"l"(p),
                 "r"(x), "r"(tag)
                 : "memory");
}

// The state words (hi, lo) of two nodes at once (the second may repeat the
// first); false when the wait gave up.
__device__ __forceinline__ bool poll_state(const float4 *xh, const float4 *xl, int g, int g0, unsigned tag, float4 &h,
                                           float4 &l, float4 &h0, int *err) {
    uint4 a = ld_word(xh + g), b = ld_word(xl + g), c = ld_word(xh + g0);
    Spin spin;
    while (a.w != tag || b.w != tag || c.w != tag) {
        if (spin.expired(err)) return false;
        if (a.w != tag) a = ld_word(xh + g);
        if (b.w != tag) b = ld_word(xl + g);
        if (c.w != tag) c = ld_word(xh + g0);
    }
    h = word_f4(a);
    l = word_f4(b);
    h0 = word_f4(c);
    return true;
}

// Control warp: |g|^2 of the instance's n CTAs, summed in double-float (each
// lane its CTAs in ascending order, then the lane tree; valid in lane 0).
__device__ __forceinline__ bool poll_r2(const uint2 *cr, int n, unsigned tag, DFloat &sum, int *err) {
    DFloat acc{0.f, 0.f};
    const int lane = threadIdx.x & 31;
    bool ok = true;
    constexpr int U = 8;
    for (int j0 = lane; j0 < n && ok; j0 += U * 32) {
        uint2 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = j0 + u * 32 < n ? ld_pair(cr + j0 + u * 32) : make_uint2(0u, tag);
        Spin spin;
        for (;;) {
            bool ready = true;
#pragma unroll
            for (int u = 0; u < U; ++u) ready &= v[u].y == tag;
            if (ready) break;
            if (spin.expired(err)) {
                ok = false;
                break;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (v[u].y != tag) v[u] = ld_pair(cr + j0 + u * 32);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (j0 + u * 32 < n) acc = df_add(acc, __uint_as_float(v[u].x));
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        acc = df_add(acc, DFloat{__shfl_down_sync(0xffffffffu, acc.hi, o), __shfl_down_sync(0xffffffffu, acc.lo, o)});
    sum = acc;
    return ok;
}

// Control warp: {sum e, sum e^2} of the instance's n CTAs in FP64, each lane
// its CTAs in ascending order, then the lane tree (valid in lane 0).  Without
// an energy slack sum e^2 scales nothing and only its finiteness matters
// (decide_line_search): it is then 0, or a NaN.
__device__ __forceinline__ bool poll_energy(const float4 *ce, int n, unsigned tag, bool slack, double &E, double &E2,
                                            int *err) {
    double a = 0.0, b = 0.0;
    bool finite = true;
    const int lane = threadIdx.x & 31;
    bool ok = true;
    constexpr int U = 4;
    for (int j0 = lane; j0 < n && ok; j0 += U * 32) {
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = j0 + u * 32 < n ? ld_word(ce + j0 + u * 32) : make_uint4(0u, 0u, 0u, tag);
        Spin spin;
        for (;;) {
            bool ready = true;
#pragma unroll
            for (int u = 0; u < U; ++u) ready &= v[u].w == tag;
            if (ready) break;
            if (spin.expired(err)) {
                ok = false;
                break;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (v[u].w != tag) v[u] = ld_word(ce + j0 + u * 32);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            a += __hiloint2double((int)v[u].y, (int)v[u].x);
            finite &= isfinite(__uint_as_float(v[u].z));
            if (slack) b += (double)__uint_as_float(v[u].z);
        }
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        if (slack) b += __shfl_down_sync(0xffffffffu, b, o);
    }
    E = a;
    E2 = slack || __all_sync(0xffffffffu, finite) ? b : __longlong_as_double(0x7ff8000000000000ll);
    return ok;
}

// A chunk's partials as tagged words.
template <int THREADS>
__device__ __forceinline__ void publish_partials(const int4 *meta, int nl, const float4 *sf, float4 *out,
                                                 unsigned tag) {
    for (int j = threadIdx.x; j < nl; j += THREADS) {
        const int4 md = meta[j];
        st_word(out + md.w, slot_sum(sf, md.y, md.z), tag);
    }
}

// The sums of a node's partials [pa, pe), in chunk order (and of its
// Jacobi-diagonal terms on a refresh pass).
__device__ __forceinline__ bool collect_partials(const DevState &st, int pa, int pe, bool do_h, unsigned tag,
                                                 NodeSums &sum, int *err) {
    constexpr int NP = 8;  // a node touches 2-8 chunks of 128-256 tets
    bool ok = true;
    for (int j = pa; j < pe; j += NP) {
        float4 f[NP];
        ok = poll_words<NP>(st.part + j, pe - j, tag, f, err) && ok;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            sum.f.x += f[q].x;
            sum.f.y += f[q].y;
            sum.f.z += f[q].z;
        }
        if (do_h) {
            ok = poll_words<NP>(st.parth + j, pe - j, tag, f, err) && ok;
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                sum.h.x += f[q].x;
                sum.h.y += f[q].y;
                sum.h.z += f[q].z;
            }
        }
    }
    return ok;
}

// What the workers need of a pass's decisions, and the next pass's decision of
// this one's update.
struct FrameView {
    int done, force_check, action;  // action: what the node update does
    float alpha, rho, omega;        // rho, omega: the pass's own (chebyshev_schedule)
};

// What a CTA owns of its instance; in shared memory, so that no register holds
// it through the tets.
struct FrameOwn {
    int n0, n1, team;  // its share of the nodes, the instance's team (at most THREADS)
};

// THREADS workers and one control warp a CTA.  A pass:
//   workers   stage the chunk's node words as they arrive, evaluate its tets,
//             publish its partials, collect the partials of their own nodes;
//   control   meanwhile collects the last pass's |g|^2 and takes its
//             decision; on a line-search pass then publishes this CTA's
//             energy, collects every CTA's and decides;
//   (one CTA barrier)
//   workers   update their nodes and publish them; warp sums of |g|^2;
//   (one CTA barrier)
//   control   publishes the CTA's |g|^2.
// The nodes of an instance are split evenly among its CTAs, in whole warps (64
// a CTA on the 24,000-tet bar), so that no CTA's node phase is longer than
// another's and the sums are the pass kernels' (phybs_internal.cuh).
// PER_SM: CTAs a SM the registers are budgeted for.  A pass is bound by the
// dependent chain of one tet, so a mesh that needs fewer CTAs a SM runs the
// variant with more registers: on 24,500 tets 493 us a 96-pass step at one
// CTA a SM (up to 246 registers, no spills), 523 at two (168: 200 bytes stored
// and 290 loaded with the full stress, 22 and 52 with the incremental, 306 and
// 408 with the stretch material), 650 at three (128: 440, 262 and 520 stored).
// For the same reason a group of 1,024 tets runs on one CTA of 256 threads,
// four tets a thread, with those 168 registers: at two CTAs a SM they have 96
// and store 608 to 780 bytes (125,000 tets: 1120 us against 855).
template <int MATERIAL, int THREADS, bool INC, bool RES, int PER_SM>
__global__ void __launch_bounds__(THREADS + 32, PER_SM)
    k_frame(DevMesh m, DevParams p, DevState st, FrameAux fx) {
    extern __shared__ float4 smem4[];
    constexpr int WARPS = THREADS / 32;
    const int CN = m.chunk_nodes, CT = m.chunk_tets;
    // node words (24 bytes a node), corner slots
    float4 *s_wa = smem4;
    float2 *s_wb = reinterpret_cast<float2 *>(smem4 + CN);
    float4 *s_f = smem4 + node_words(CN, INC, 0);
    // resident: the chunk's rows and records
    float4 *s_r0 = s_f + m.chunk_slots, *s_r1 = s_r0 + CT, *s_r2 = s_r1 + CT;
    uint4 *s_cor = reinterpret_cast<uint4 *>(s_r2 + CT);
    int4 *s_meta = reinterpret_cast<int4 *>(s_cor + CT);
    __shared__ InstCtl sc;  // this CTA's copy of the instance's control block (the control warp's)
    __shared__ FrameView sv;
    __shared__ FrameOwn own;
    __shared__ float2 s_e[WARPS];
    __shared__ float s_e2[WARPS], s_g2[SUM_GROUPS];
    const int b = blockIdx.x, tid = threadIdx.x;
    const bool worker = tid < THREADS;
    const int inst = RES ? m.chunk_inst[b] : 0;
    if (tid == 0) sc = st.ctl[inst];
    if (RES && worker) {
        const int4 cd = m.chunk[b];
        for (int t = tid; t < cd.y; t += THREADS) {
            cp_async16(s_r0 + t, m.qrow0 + cd.x + t);
            cp_async16(s_r1 + t, m.qrow1 + cd.x + t);
            cp_async16(s_r2 + t, m.qrow2 + cd.x + t);
            cp_async16(s_cor + t, m.qcor + cd.x + t);
        }
        for (int j = tid; j < cd.w; j += THREADS) {
            const int4 md = m.lmeta[cd.z + j];
            s_meta[j] = md;
            if (INC) pack_words(s_wa, s_wb, j, st.ub[md.x], st.ub[md.x]);  // (the base; the increment follows)
        }
        cp_async_commit();
        cp_async_wait_all();
    }
    __syncthreads();
    if (sc.done) return;  // an instance without tets or iterations: none of its CTAs waits
    const int cb = RES ? sc.cblk_begin : 0;
    const int G = RES ? sc.cblk_end - cb : (int)gridDim.x;  // CTAs of the instance, this one bi
    const int bi = b - cb;
    int *err = st.active + 1;
    // this CTA's nodes [n0, n1), this thread's i0, i0 + THREADS, ...
    if (tid == 0) {
        const int per = node_share(sc.node_end - sc.node_begin, G);
        own.n0 = min(sc.node_begin + bi * per, sc.node_end);
        own.n1 = min(own.n0 + per, sc.node_end);
        own.team = RES ? sc.team : THREADS;
    }
    __syncthreads();
    // (the variant with registers to spare keeps its nodes in them)
    constexpr bool REGS = THREADS == 128 && PER_SM == 1;
    const int rn0 = own.n0, rn1 = own.n1;
    auto n0 = [&] { return REGS ? rn0 : own.n0; };
    auto n1 = [&] { return REGS ? rn1 : own.n1; };
    auto team = [&] { return THREADS == 128 ? 128 : own.team; };  // (no team is smaller than 128)
    // this thread's first node is n0() + tid: mine() whether it has one
    auto mine = [&] { return worker && n0() + tid < n1(); };
    int pa0 = 0, pe0 = 0;
    if (mine()) {
        pa0 = m.pptr[n0() + tid];
        pe0 = m.pptr[n0() + tid + 1];
    }
    int k = sc.k, par = sc.par;
    bool force = sc.force_check != 0;
    {
        const size_t cur = (size_t)par * m.Np;
        for (int i = n0() + tid; worker && i < n1(); i += THREADS) {
            const float4 h = st.uh[cur + i], l = st.ul[cur + i];
            st_word(fx.xh + i, make_float3(h.x, h.y, h.z), fx.tag0 + 1);
            st_word(fx.xl + i, make_float3(l.x, l.y, l.z), fx.tag0 + 1);
        }
    }
    __syncthreads();    // sc is the control warp's from here
    bool ok = true;     // no wait of this thread gave up
    bool pend = false;  // the pass decision of the last node update is not taken yet
    for (int pass = 0;;) {
        const unsigned tag = fx.tag0 + 1 + (unsigned)pass;
        // the pass runs on the foreseen outcome of the pending decision
        const size_t cur = (size_t)par * m.Np;
        const bool check = (k % p.ls_every) == 0 || force;
        const bool do_h = (k % p.hd_every) == 0;
        // a run's last update (pbs_profile_frame) is only settled
        const bool last = pass >= fx.max_passes;
        NodeConst nc;
        NodeIn nn;
        NodeSums sum{make_float3(0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f)};
        if (worker && !last) {
            DFloat e{0.f, 0.f};
            float e2 = 0.f;
            // the words of this thread's first node, only ever written by itself
            if (mine()) {
                const int i0 = n0() + tid;
                nn.uh = st.uh[cur + i0];
                nn.ul = st.ul[cur + i0];
                nn.dd = st.dd[cur + i0];
                nn.diag = st.diag[i0];
            }
            // the CTA's share of the node energy terms, before the other CTAs'
            // words arrive
            if (check && tid < team())
                share_energy(m, p, st, cur, n0() + tid, n1(), team(), INC ? st.ub : nullptr, e, e2);
            // ---- tet phase: this CTA's chunk, or the chunks b, b + G, ...
            for (int c = b; c < m.n_chunks; c += RES ? m.n_chunks : G) {
                const int4 cd = m.chunk[c];
                const int nt = cd.y, nl = cd.w;
                const int4 *meta = RES ? s_meta : m.lmeta + cd.z;
                const int g0 = nl ? meta[0].x : 0;
                for (int j = tid; j < nl; j += THREADS) {
                    const int g = meta[j].x;
                    float4 uh, ul, r;  // (the increments relative to the chunk's local node 0)
                    ok = poll_state(fx.xh, fx.xl, g, INC ? g0 : g, tag, uh, ul, r, err) && ok;
                    if (!INC) {
                        pack_words(s_wa, s_wb, j, uh, ul);
                    } else if (RES) {  // the base is there already
                        const float4 d = increment_rel(uh, ul, r);
                        s_wa[j].x = d.x;
                        s_wa[j].y = d.y;
                        s_wa[j].z = d.z;
                    } else {
                        pack_words(s_wa, s_wb, j, increment_rel(uh, ul, r), st.ub[g]);
                    }
                }
                if (c == b && pend) asm volatile("barrier.cta.arrive 2, %0;" ::"n"(THREADS + 32) : "memory");
                chunk_sync<THREADS, true>();
                ChunkView v;
                v.wa = s_wa;
                v.wb = s_wb;
                v.r0 = RES ? s_r0 : m.qrow0 + cd.x;
                v.r1 = RES ? s_r1 : m.qrow1 + cd.x;
                v.r2 = RES ? s_r2 : m.qrow2 + cd.x;
                v.cor = RES ? s_cor : m.qcor + cd.x;
                v.meta = meta;
                v.rest = m.rest;
                DFloat ec = chunk_forces_all<MATERIAL, THREADS, INC, true, false, true>(p, v, nt, check, s_f);
                if (check && team() != THREADS && tid < team()) ec = team_energy(v.cor, nt, tid, team(), s_f);
                publish_partials<THREADS>(meta, nl, s_f, st.part, tag);
                if (do_h) {
                    chunk_sync<THREADS, true>();
                    chunk_hdiag<MATERIAL, THREADS, INC, true>(v, nt, s_f);
                    chunk_sync<THREADS, true>();
                    publish_partials<THREADS>(meta, nl, s_f, st.parth, tag);
                }
                if (check && tid < team()) {
                    e = df_add(e, ec);
                    e2 += noise_square(m, team(), nt, ec.hi);
                }
                // the slots and node words are free for the next chunk (or pass)
                if (!RES) chunk_sync<THREADS, true>();
            }
            if (check) {
                e = warp_sum_df(e);
                e2 = warp_sum_f(e2);
                if ((tid & 31) == 0) {
                    s_e[tid >> 5] = make_float2(e.hi, e.lo);
                    s_e2[tid >> 5] = e2;
                }
            }
        }
        // ---- the pass decision (every CTA's control warp, the same words)
        if (!worker && pend) {
            // not before this CTA's node words have arrived: the |g|^2 words
            // then have too, where polling them from every CTA at once slowed
            // the other exchanges (8.0 against 6.3 us a pass with 196 CTAs)
            if (!last) asm volatile("barrier.cta.sync 2, %0;" ::"n"(THREADS + 32) : "memory");
            DFloat R;
            ok = poll_r2(fx.cr + ((pass - 1) & 1) * gridDim.x + cb, G, tag - 1, R, err);
            if (tid == THREADS) {
                decide_pass(sc, p, sc.k, sv.action, sv.rho, sv.omega, df_double(R));
                // (settle_pass's count of a void pass)
                if (fx.count_void && !last && !sc.done && sc.force_check && !check && ++sc.passes >= p.pass_cap) {
                    sc.done = 1;
                    sc.status = PBS_E_ITER_CAP;
                }
            }
            __syncwarp();
        }
        if (check && !last) {
            // ---- line search: this CTA's energy, then the decision from every
            // CTA's
            __syncthreads();
            if (!worker && !sc.done) {
                double d;
                float se2;
                join_warps(s_e, s_e2, team(), d, se2);
                if (tid == THREADS)
                    st_word(fx.ce + b, (unsigned)__double2loint(d), (unsigned)__double2hiint(d),
                            __float_as_uint(se2), tag);
                __syncwarp();
                double E, E2;
                ok = poll_energy(fx.ce + cb, G, tag, p.energy_slack != 0.f, E, E2, err) && ok;
                if (tid == THREADS) decide_line_search(sc, p, k, E, E2);
            }
        }
        if (!worker) {
            if (tid == THREADS) {
                sv.done = sc.done;
                sv.force_check = sc.force_check;
                sv.action = check ? sc.action : ACT_STEP;
                sv.alpha = sc.alpha;
                float r = sc.rho, o = sc.omega;
                chebyshev_schedule(p, k - sc.k_restart, r, o);
                sv.rho = r;
                sv.omega = o;
            }
        } else if (!last && mine()) {
            // the partials of this thread's first node.  Every partial is
            // waited for whether or not the update needs it (pinned nodes, a
            // restore): the chunks have then read the state word that the
            // update overwrites
            nc.ch = st.ch[n0() + tid];
            nc.cl = st.cl[n0() + tid];
            ok = collect_partials(st, pa0, pe0, do_h, tag, sum, err) && ok;
        }
        ok = !__syncthreads_or(!ok);
        if (!ok) break;
        pend = false;
        if (sv.done || last) break;
        if (sv.force_check && !check) {
            force = true;  // the energy check the decision forces: this pass again
            __syncthreads();
            continue;
        }
        // ---- node phase
        force = false;
        PassCtx ctx;
        ctx.action = sv.action;
        ctx.do_h = do_h;
        ctx.alpha = sv.alpha;
        ctx.omega = sv.omega;
        ctx.cur = cur;
        ctx.nxt = (size_t)(1 - par) * m.Np;
        // (by whole warps: a warp's nodes are one group of 32)
        for (int g = tid & ~31; worker && g < n1() - n0(); g += THREADS) {
            const int i = n0() + g + (tid & 31);
            float r2 = 0.f;
            if (i < n1()) {
                if (g >= THREADS) {
                    nc.ch = st.ch[i];
                    nc.cl = st.cl[i];
                    nn.uh = st.uh[cur + i];
                    nn.ul = st.ul[cur + i];
                    nn.dd = st.dd[cur + i];
                    nn.diag = st.diag[i];
                    sum = NodeSums{make_float3(0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f)};
                    ok = collect_partials(st, m.pptr[i], m.pptr[i + 1], do_h, tag, sum, err) && ok;
                }
                float4 x[2];
                r2 = node_update(p, st, i, nc, nn, ctx, [&] { return sum; }, x);
                st_word(fx.xh + i, make_float3(x[0].x, x[0].y, x[0].z), tag + 1);
                st_word(fx.xl + i, make_float3(x[1].x, x[1].y, x[1].z), tag + 1);
            }
            r2 = warp_sum_f(r2);
            // (beyond SUM_GROUPS groups the same warp's places again)
            float *o = s_g2 + (g >> 5) % SUM_GROUPS;
            if ((tid & 31) == 0) *o = (g >> 5) < SUM_GROUPS ? r2 : *o + r2;
        }
        __syncthreads();
        if (tid == THREADS) {
            float s = 0.f;
            const int groups = min((n1() - n0() + 31) >> 5, SUM_GROUPS);
            for (int g = 0; g < groups; g += WARPS) {
                float v[WARPS];
#pragma unroll
                for (int w = 0; w < WARPS; ++w) v[w] = g + w < groups ? s_g2[g + w] : 0.f;
#pragma unroll
                for (int w = 0; w < WARPS; ++w) s += v[w];
            }
            st_pair(fx.cr + (pass & 1) * gridDim.x + b, __float_as_uint(s), tag);
        }
        __syncwarp();
        pend = true;
        if (sv.action != ACT_RESTORE) ++k;
        par ^= 1;
        ++pass;
    }
    if (bi == 0 && tid == THREADS) {
        if (!ok) {
            sc.status = PBS_E_DEVICE_TIMEOUT;
            sc.done = 1;
        }
        st.ctl[inst] = sc;
        if (sc.done) atomicSub(st.active, 1);
    }
}

// Shared memory of a CTA: the pass kernel's node words and slots, with the
// resident layout also the rows and records.
static size_t frame_smem(const DevMesh &m, bool inc, bool resident) {
    return chunk_smem(m.chunk_tets, m.chunk_nodes, m.chunk_slots, inc, 0) +
           (resident ? 64 * (size_t)m.chunk_tets + sizeof(int4) * (size_t)m.chunk_nodes : 0);
}

// Co-resident CTAs of a variant on a device with `sms` SMs.
template <int MATERIAL, int THREADS, bool INC, bool RES, int PER_SM>
static int frame_fit(const DevMesh &m, int sms) {
    const auto kernel = k_frame<MATERIAL, THREADS, INC, RES, PER_SM>;
    const size_t smem = frame_smem(m, INC, RES);
    int per_sm = 0;
    if (smem > (size_t)CHUNK_MAX_SMEM ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CHUNK_MAX_SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, THREADS + 32, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return per_sm * sms;
}

template <int MATERIAL, int THREADS, bool INC, bool RES, int PER_SM>
static cudaError_t launch_frame_v(cudaStream_t s, const DevMesh &m, const DevParams &p, const DevState &st,
                                  const FrameAux &fx, int grid) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(THREADS + 32);
    cfg.dynamicSmemBytes = frame_smem(m, INC, RES);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_frame<MATERIAL, THREADS, INC, RES, PER_SM>, m, p, st, fx);
}

// The register classes: resident 128-thread CTAs at one, two or three a SM,
// 256-thread CTAs at one or two; walking five and three.
template <int MATERIAL, int THREADS, bool INC>
static cudaError_t launch_frame_t(cudaStream_t s, const DevMesh &m, const DevParams &p, const DevState &st,
                                  const FrameAux &fx, const FramePlan &plan) {
    constexpr int WALK = THREADS == 128 ? 5 : 3;
    if (!plan.resident) return launch_frame_v<MATERIAL, THREADS, INC, false, WALK>(s, m, p, st, fx, plan.grid);
    if (plan.per_sm == 1) return launch_frame_v<MATERIAL, THREADS, INC, true, 1>(s, m, p, st, fx, plan.grid);
    if constexpr (THREADS == 128) {
        if (plan.per_sm == 3) return launch_frame_v<MATERIAL, 128, INC, true, 3>(s, m, p, st, fx, plan.grid);
    }
    return launch_frame_v<MATERIAL, THREADS, INC, true, 2>(s, m, p, st, fx, plan.grid);
}

template <int MATERIAL, int THREADS, bool INC> static FramePlan frame_plan_t(const DevMesh &m, int sms) {
    constexpr int WALK = THREADS == 128 ? 5 : 3;
    FramePlan r;
    r.resident = true;
    r.grid = m.n_chunks;
    r.per_sm = 1;
    if (frame_fit<MATERIAL, THREADS, INC, true, 1>(m, sms) >= m.n_chunks) return r;
    r.per_sm = 2;
    if (frame_fit<MATERIAL, THREADS, INC, true, 2>(m, sms) >= m.n_chunks) return r;
    if constexpr (THREADS == 128) {
        r.per_sm = 3;
        if (frame_fit<MATERIAL, 128, INC, true, 3>(m, sms) >= m.n_chunks) return r;
    }
    r = FramePlan{};
    if (m.n_inst == 1) r.grid = std::min(m.n_chunks, frame_fit<MATERIAL, THREADS, INC, false, WALK>(m, sms));
    return r;
}

// material / stress / thread-count dispatch of f<MATERIAL, THREADS, INC>
#define PBS_FRAME_DISPATCH(f, ...)                                                                        \
    (material == PBS_MATERIAL_STRETCH                                                                     \
         ? (m.chunk_threads == 128 ? f<PBS_MATERIAL_STRETCH, 128, false>(__VA_ARGS__)                     \
                                   : f<PBS_MATERIAL_STRETCH, 256, false>(__VA_ARGS__))                    \
         : inc ? (m.chunk_threads == 128 ? f<PBS_MATERIAL_NEOHOOKEAN, 128, true>(__VA_ARGS__)             \
                                         : f<PBS_MATERIAL_NEOHOOKEAN, 256, true>(__VA_ARGS__))            \
               : (m.chunk_threads == 128 ? f<PBS_MATERIAL_NEOHOOKEAN, 128, false>(__VA_ARGS__)            \
                                         : f<PBS_MATERIAL_NEOHOOKEAN, 256, false>(__VA_ARGS__)))

FramePlan frame_plan(const DevMesh &m, int material, bool inc, int sms) {
    if (m.chunk_stage != 0 || m.n_chunks <= 0 || (m.chunk_threads != 128 && m.chunk_threads != 256))
        return FramePlan{};
    return PBS_FRAME_DISPATCH(frame_plan_t, m, sms);
}

cudaError_t launch_frame(cudaStream_t s, const DevMesh &m, const DevParams &p, DevState st, int material,
                         const FrameAux &fx, const FramePlan &plan) {
    if (plan.grid <= 0) return cudaErrorInvalidConfiguration;
    const bool inc = material == PBS_MATERIAL_NEOHOOKEAN && p.incremental;
    return PBS_FRAME_DISPATCH(launch_frame_t, s, m, p, st, fx, plan);
}

}  // namespace pbs

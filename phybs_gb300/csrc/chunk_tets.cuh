// The tets of one chunk in a descent pass: corner forces into shared-memory
// slots, the slots' sums into per-(node, chunk) partials, the Jacobi diagonal.
// Shared by the pass kernels of the graph path (chunks.cu) and the persistent
// frame kernel (frame.cu).
#pragma once
#include "../../include/phybs.h"
#include "pass_math.cuh"
#include "phybs_internal.cuh"
#include "tet_math.cuh"

namespace pbs {

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Corner ids of a pass tet from its packed record.
__device__ __forceinline__ void unpack_cor(const uint4 &w, int loc[4], int slot[4]) {
    loc[0] = (int)(w.x & 0xffffu);
    loc[1] = (int)(w.x >> 16);
    loc[2] = (int)(w.y & 0xffffu);
    loc[3] = (int)(w.y >> 16);
    slot[0] = (int)(w.z & 0xffffu);
    slot[1] = (int)(w.z >> 16);
    slot[2] = (int)(w.w & 0xffffu);
    slot[3] = (int)(w.w >> 16);
}

// One chunk as its tet loop reads it: node words staged in shared memory;
// per-tet rows and corner records in shared memory or at the chunk's place in
// the pass arrays.
//
// A local node's words are two vectors: its displacement u (hi, lo; full
// stress), or its increment relative to the chunk's reference node and its
// base (incremental stress).  PACK: the six floats as {v0, v1.x} in wa and
// {v1.y, v1.z} in wb, 24 bytes: the tet loop is bound by its shared-memory
// wavefronts (64% of the active cycles on the 512,000-tet box), and two
// 128-bit words a node, a quarter of them unused, were a third of those.
// Otherwise (rows staged by asynchronous copies, which bring 16-byte words) as
// float4 in uh / ul / ub.
struct ChunkView {
    float4 *wa;
    float2 *wb;
    const float4 *uh, *ul, *ub;
    const float4 *r0, *r1, *r2;
    const uint4 *cor;
    const int4 *meta;    // local-node records (their global ids locate the rest positions)
    const float4 *rest;  // rest positions, for the FP64 stress of a near-inverted tet
};

// Stores local node j's words (PACK): v0 = u hi or the increment, v1 = u lo or
// the base.
__device__ __forceinline__ void pack_words(float4 *wa, float2 *wb, int j, const float4 &v0, const float4 &v1) {
    wa[j] = make_float4(v0.x, v0.y, v0.z, v1.x);
    wb[j] = make_float2(v1.y, v1.z);
}

// The node words of a tet's four corners: x = u hi (full stress) or nothing
// (the incremental form), l = u lo or the increment relative to the chunk's
// reference node, a = the base (incremental).
template <bool INC, bool PACK>
__device__ __forceinline__ void corner_words(const ChunkView &v, const int lc[4], float4 x[4], float4 l[4],
                                             float4 a[4]) {
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (PACK) {
            const float4 p = lds128(v.wa + lc[c]);
            const float2 q = lds64(v.wb + lc[c]);
            const float4 v0 = make_float4(p.x, p.y, p.z, 0.f), v1 = make_float4(p.w, q.x, q.y, 0.f);
            x[c] = INC ? z4 : v0;
            l[c] = INC ? v0 : v1;
            a[c] = INC ? v1 : z4;
        } else {
            x[c] = INC ? z4 : lds128(v.uh + lc[c]);
            l[c] = lds128(v.ul + lc[c]);
            a[c] = INC ? lds128(v.ub + lc[c]) : z4;
        }
    }
}

// A tet's constants.
struct TetRows {
    float4 r0, r1, r2;
    uint4 cor;
};
__device__ __forceinline__ TetRows load_rows(const ChunkView &v, int lt) {
    return TetRows{v.r0[lt], v.r1[lt], v.r2[lt], v.cor[lt]};
}

// Corner forces of the chunk's tets into the slots; on line-search passes
// returns the thread's sum of clamped tet energies.
// A near-inverted tet (full stress) gets its FP32 forces here and a mark in
// its corner-0 slot's .w; *any_exact tells whether the thread marked one.
// CHECK: a line-search pass (the tet energies too, each also in its corner-1
// slot's .w for team_energy); the loop is compiled once with and once without
// them.  first: the constants of the thread's first tet,
// where the caller loaded them ahead (PRE).
template <int MATERIAL, int THREADS, bool INC, bool PACK, bool PRE, bool CHECK>
__device__ __forceinline__ DFloat chunk_forces(const DevParams &p, const ChunkView &v, int nt, float4 *sf,
                                               bool *any_exact, const TetRows &first) {
    DFloat e{0.f, 0.f};
    bool any = false;
    TetRows rows = first;
    for (int lt = threadIdx.x; lt < nt; lt += THREADS) {
        if (!PRE || lt != threadIdx.x) rows = load_rows(v, lt);
        const float4 r0 = rows.r0, r1 = rows.r1, r2 = rows.r2;
        int lc[4], sl[4];
        unpack_cor(rows.cor, lc, sl);
        const float dinv[9] = {r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r2.x, r2.y, r2.z};
        Kin<float> kin;
        float f[12];
        float4 x[4], l[4], a[4];
        corner_words<INC, PACK>(v, lc, x, l, a);
        const bool ex = pass_forces_c<MATERIAL, INC, true, CHECK>(
            x[0], x[1], x[2], x[3], l[0], l[1], l[2], l[3], a[0], a[1], a[2], a[3], dinv, r0.w, r1.w, r2.w, kin, f,
            CornerRest{v.rest, v.meta, {lc[0], lc[1], lc[2], lc[3]}});
        any |= ex;
#pragma unroll
        for (int cc = 0; cc < 4; ++cc)
            sts128(sf + sl[cc], f[3 * cc], f[3 * cc + 1], f[3 * cc + 2], cc == 0 && ex ? 1.f : 0.f);
        if (CHECK) {
            const float en = search_energy(energy_density<float>(kin, r1.w, r2.w) * fabsf(r0.w), p.clamp_cpu,
                                           p.control == PBS_CONTROL_RESTART);
            e = df_add(e, en);
            sf[sl[1]].w = en;
        }
    }
    *any_exact = any;
    return e;
}

// The stretch-based stress from the FP32 SVD; false where it is too
// ill-conditioned (near inversion, or sigma_3 < 0.3).  Out of line: few tets
// take it.
static __device__ __noinline__ bool chunk_stretch_svd(const float4 x[4], const float4 l[4], const float dinv[9],
                                                      float mu, float lambda, float P[9]) {
    Kin<float> kin;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    disp_gradient<float>(z, f4add(f4sub(x[1], x[0]), f4sub(l[1], l[0])), f4add(f4sub(x[2], x[0]), f4sub(l[2], l[0])),
                         f4add(f4sub(x[3], x[0]), f4sub(l[3], l[0])), dinv, kin.G);
    kinematics(kin);
    return 1.0f + kin.d >= 1e-3f && stretch_pk1<float>(kin.G, mu, lambda, P);
}

// The FP64 stress of the chunk's marked (near-inverted) tets, into their
// slots.  After the tet loop rather than inside it: the loop then carries no
// call, and keeps its registers.
template <int MATERIAL, int THREADS, bool PACK>
__device__ __forceinline__ void chunk_exact(const ChunkView &v, int nt, float4 *sf) {
    for (int lt = threadIdx.x; lt < nt; lt += THREADS) {
        int lc[4], sl[4];
        unpack_cor(v.cor[lt], lc, sl);
        if (lds128(sf + sl[0]).w == 0.f) continue;
        const float4 r0 = v.r0[lt], r1 = v.r1[lt], r2 = v.r2[lt];
        const float dinv[9] = {r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r2.x, r2.y, r2.z};
        float4 x[4], l[4], a[4];
        corner_words<false, PACK>(v, lc, x, l, a);
        float P[9], f[12];
        // a stretch-material tet that only may be ill-conditioned: the FP32
        // SVD decides
        if (MATERIAL != PBS_MATERIAL_STRETCH || !chunk_stretch_svd(x, l, dinv, r1.w, r2.w, P))
            pk1_exact_fp64(MATERIAL, CornerRest{v.rest, v.meta, {lc[0], lc[1], lc[2], lc[3]}}, x[0], x[1], x[2],
                           x[3], l[0], l[1], l[2], l[3], r0, r1, r2, r1.w, r2.w, P);
        corner_forces(P, dinv, r0.w, f);
        const float en = lds128(sf + sl[1]).w;
#pragma unroll
        for (int cc = 0; cc < 4; ++cc)
            sts128(sf + sl[cc], f[3 * cc], f[3 * cc + 1], f[3 * cc + 2], cc == 1 ? en : 0.f);
    }
}

// Barrier of the threads that evaluate a chunk: the whole CTA, or (PART) its
// first THREADS threads on a barrier of their own.
template <int THREADS, bool PART> __device__ __forceinline__ void chunk_sync() {
    if (PART) asm volatile("barrier.cta.sync 1, %0;" ::"n"(THREADS) : "memory");
    else __syncthreads();
}
template <int THREADS, bool PART> __device__ __forceinline__ bool chunk_sync_or(bool x) {
    if (!PART) return __syncthreads_or(x) != 0;
    unsigned r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((unsigned)x), "n"(THREADS)
        : "memory");
    return r != 0;
}

// chunk_forces, then the FP64 stress of a chunk that has a near-inverted tet;
// every (participating) thread sees the finished slots on return.
template <int MATERIAL, int THREADS, bool INC, bool PACK, bool PRE, bool PART = false>
__device__ __forceinline__ DFloat chunk_forces_all(const DevParams &p, const ChunkView &v, int nt, bool check,
                                                   float4 *sf, const TetRows &first = TetRows()) {
    bool ex;
    const DFloat e = check ? chunk_forces<MATERIAL, THREADS, INC, PACK, PRE, true>(p, v, nt, sf, &ex, first)
                           : chunk_forces<MATERIAL, THREADS, INC, PACK, PRE, false>(p, v, nt, sf, &ex, first);
    if (INC) {
        chunk_sync<THREADS, PART>();
    } else if (chunk_sync_or<THREADS, PART>(ex)) {
        chunk_exact<MATERIAL, THREADS, PACK>(v, nt, sf);
        chunk_sync<THREADS, PART>();
    }
    return e;
}

// Thread t's sum of a piece's tet energies where the tet loop did not form it
// (the instance's team is not the CTA's threads, or the chunk has several
// pieces): the tets t, t + team, ... of the nt whose corner records start at
// cor, from the slots that the tet loop left them in.  Before anything else
// goes into the slots.
__device__ __forceinline__ DFloat team_energy(const uint4 *cor, int nt, int t, int team, const float4 *sf) {
    DFloat e{0.f, 0.f};
    for (int lt = t; lt < nt; lt += team) {
        int lc[4], sl[4];
        unpack_cor(cor[lt], lc, sl);
        e = df_add(e, lds128(sf + sl[1]).w);
    }
    return e;
}

// The energy terms of the nodes [n, n1), every team-th, added to the thread's e
// and their squares to e2.
__device__ __forceinline__ void share_energy(const DevMesh &m, const DevParams &p, const DevState &st, size_t cur, int n,
                                             int n1, int team, const float4 *base, DFloat &e, float &e2) {
    for (int i = n; i < n1; i += team) {
        const float4 info = m.info[i];
        if (info.z != 0.f) continue;
        const DFloat en = node_energy_df(st, info, st.uh[cur + i], st.ul[cur + i], i, p.h2inv, base);
        e = df_add(e, en);
        e2 = fmaf(en.hi, en.hi, e2);
    }
}

// A thread's share of the line search's noise scale, from the sum e of its tet
// energies: the scale adds the squares of the sums of m.noise_tets tets (four,
// whose threads' sums are grouped by neighbouring lanes; 0: of each thread's
// own), so that a line search rejects by the same allowance at every automatic
// chunk size.  With each thread's own at one or two tets a thread the allowance
// was half as large, and one pull in ten to a residual of 1e-4 took another
// rejection.  Called by whole warps.
__device__ __forceinline__ float noise_square(const DevMesh &m, int team, int nt, float e) {
    const int lanes = m.noise_tets == 0 || nt > 3 * team ? 1 : nt > team ? m.noise_tets / 2 : m.noise_tets;
    if (lanes > 1) e += __shfl_xor_sync(0xffffffffu, e, 1);
    if (lanes > 2) e += __shfl_xor_sync(0xffffffffu, e, 2);
    return e * e / (float)lanes;
}

// A chunk's sums from the warps' (s_e, s_e2: team / 32 of them), by one warp;
// valid in lane 0.
__device__ __forceinline__ void join_warps(const float2 *s_e, const float *s_e2, int team, double &e, float &e2) {
    const int warps = team >> 5, w = threadIdx.x & (warps - 1);
    DFloat se{s_e[w].x, s_e[w].y};
    e2 = s_e2[w];
    for (int o = warps >> 1; o > 0; o >>= 1) {
        se = df_add(se, DFloat{__shfl_down_sync(0xffffffffu, se.hi, o), __shfl_down_sync(0xffffffffu, se.lo, o)});
        e2 += __shfl_down_sync(0xffffffffu, e2, o);
    }
    e = df_double(se);
}

// Jacobi-diagonal refresh: the same slots carry the 12 diagonal terms.
template <int MATERIAL, int THREADS, bool INC, bool PACK>
__device__ __forceinline__ void chunk_hdiag(const ChunkView &v, int nt, float4 *sf) {
    for (int lt = threadIdx.x; lt < nt; lt += THREADS) {
        const float4 r0 = v.r0[lt], r1 = v.r1[lt], r2 = v.r2[lt];
        int lc[4], sl[4];
        unpack_cor(v.cor[lt], lc, sl);
        const float dinv[9] = {r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r2.x, r2.y, r2.z};
        Kin<float> kin;
        float f[12], kd[12];
        float4 x[4], l[4], a[4];
        corner_words<INC, PACK>(v, lc, x, l, a);
        // only the kinematics are used here (no FP64 stress needed)
        pass_forces_c<MATERIAL, INC, true>(x[0], x[1], x[2], x[3], l[0], l[1], l[2], l[3], a[0], a[1], a[2], a[3],
                                           dinv, r0.w, r1.w, r2.w, kin, f,
                                           CornerRest{v.rest, v.meta, {lc[0], lc[1], lc[2], lc[3]}});
        hessian_diag(kin, r1.w, r2.w, dinv, r0.w, kd);
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) sts128(sf + sl[cc], kd[3 * cc], kd[3 * cc + 1], kd[3 * cc + 2]);
    }
}

// The sum of a local node's slots, in slot order.  The slots are read four at
// a time ahead of their additions: one shared-memory round trip a slot was
// half of the partial sums' time.
__device__ __forceinline__ float3 slot_sum(const float4 *sf, int s, int e) {
    float3 a = make_float3(0.f, 0.f, 0.f);
    for (; s + 4 <= e; s += 4) {
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = lds128(sf + s + u);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            a.x += q[u].x;
            a.y += q[u].y;
            a.z += q[u].z;
        }
    }
    for (; s < e; ++s) {
        const float4 q = lds128(sf + s);
        a.x += q.x;
        a.y += q.y;
        a.z += q.z;
    }
    return a;
}

// Sums every local node's slots into its partial for this chunk.  meta: the
// chunk's local-node records (shared or global memory).
template <int THREADS>
__device__ __forceinline__ void chunk_partials(const int4 *meta, int nl, const float4 *sf, float4 *out) {
    for (int j = threadIdx.x; j < nl; j += THREADS) {
        const int4 md = meta[j];
        const float3 a = slot_sum(sf, md.y, md.z);
        out[md.w] = make_float4(a.x, a.y, a.z, 0.f);
    }
}

}  // namespace pbs

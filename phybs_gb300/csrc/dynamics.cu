// The reference's two other CPU integrators, on the device:
//
// Strain-based position-based dynamics (PosBaseDynamic.cpp:12-117, Mueller et
// al. 2014): Gauss-Seidel sweeps over the tets in the caller's order.  A
// serial sweep is reproduced exactly by dependency levels: a tet's level is
// one more than the highest level of the earlier tets that share one of its
// nodes, so a level's tets share no node and each reads exactly the updates of
// the tets before it in the serial order.  One thread-block cluster sweeps an
// instance step by step (16 CTAs when the handle holds few instances, else
// 8), a step being one level of each sweep in flight (PbdStep), the cluster
// barrier ordering the steps (its arrive/wait carry release/acquire semantics
// for the positions): 2,496 steps of up to 2,150 tets for five sweeps of the
// 1M-tet box (2,320 levels), 636 for the 24K bar (348 levels).  The
// arithmetic is FP32 with every product and sum rounded separately (no
// contraction) in Eigen 3.2's order, so a sweep is the CPU's bit for bit.
//
// Projective dynamics (ProjDynamic.cpp:48-100, 351-480): per-tet polar
// rotations from the modified SVD and the constant global matrix A = L (x) I3.
// A p and b are of the size of the positions times the stiffness, and an
// FP32 A's rows do not sum to zero exactly, so applied to absolute positions
// it would add forces proportional to the distance from the origin.  Each
// global solve is therefore a correction from a residual formed without
// absolute coordinates: r = b - A p = M / dt^2 ((x - p) + q) +
// sum_t k vol (R - F) w_a (edge differences only), A d = r by the
// block-Jacobi conjugate gradients of the backward-Euler step, p += d.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "../../include/phybs.h"
#include "phybs_internal.cuh"
#include "tet_math.cuh"

namespace cg = cooperative_groups;

namespace pbs {

namespace {

// CTAs a PBD cluster sweeps an instance with: 16 (the non-portable maximum,
// opted into at launch) when a handle holds few instances, else 8
constexpr int kPbdClusterMax = 16;
// worker threads of a CTA, and the scheduler warp: the eighth, whose warp
// scheduler the first seven leave to at most one other
constexpr int kPbdWorkers = 224;
constexpr int kPbdThreads = kPbdWorkers + 32;

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
// Eigen 3.2's 3-vector dot / squaredNorm: x0 + (x1 + x2)
__device__ __forceinline__ float dot3e(const float a[3], const float b[3]) {
    return fadd(fmul(a[0], b[0]), fadd(fmul(a[1], b[1]), fmul(a[2], b[2])));
}

// float(((double)S - 1.0) / (double)lam * (double)k): the reference's stretch
// multiplier, whose double literal makes it FP64 (PosBaseDynamic.cpp:100).
// GB300's FP64 pipe is narrow, so the value is formed in double-float FP32
// (error below 2^-44 relative) and rounded; the FP64 expression is evaluated
// only when that value lies within 2^-40 relative of a float rounding
// boundary, where the two roundings could differ (or for zero, non-finite or
// tiny values).  Published methods used: the quotient is Markstein's
// correction of an approximate reciprocal by its exact FMA remainder
// r = a - q b (P. Markstein, "IA-64 and Elementary Functions", 2000, ch. 8);
// S - 1 and the product by k use the error-free transformations TwoSum
// (Knuth, TAOCP vol. 2, 4.2.2) and the FMA form of TwoProduct (Ogita, Rump
// and Oishi, "Accurate sum and dot product", SIAM J. Sci. Comput. 26, 2005),
// and the final renormalisation is Dekker's FastTwoSum (Dekker, Numer. Math.
// 18, 1971).  The boundary test then decides whether the double-float value
// determines the FP32 rounding of the exact FP64 quotient.
__device__ __forceinline__ float pbd_stretch_mult(float S, float lam, float k) {
    float ah, al;
    two_sum(S, -1.0f, ah, al);  // S - 1 = ah + al exactly
    if (ah == 0.0f && al == 0.0f) return fmul(0.0f, k);
    // (ah + al) / lam as q1 + q2 from one approximate reciprocal: q1 is within
    // a few ulp, the remainder ah - q1 lam is formed by one fma (exact, or
    // rounded at 2^-24 of itself) and corrected by q2; |error| < 2^-45 of the
    // quotient, well inside the boundary test's 2^-40 margin below
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(lam));
    const float q1 = fmul(ah, inv);
    const float r = fadd(__fmaf_rn(-q1, lam, ah), al);
    const float q2 = fmul(r, inv);
    const float p1 = fmul(q1, k);
    const float p2 = __fmaf_rn(q2, k, __fmaf_rn(q1, k, -p1));  // q1 k - p1 is exact
    const float c = fadd(p1, p2);
    const float d = fadd(fsub(p1, c), p2);  // (p1 + p2) - c
    const float ac = fabsf(c);
    if (ac < 1e-30f || ac > 1e30f || !isfinite(ac))
        return __double2float_rn(__dmul_rn(__ddiv_rn(__dsub_rn((double)S, 1.0), (double)lam), (double)k));
    // the float boundary on d's side of c: half the gap to the neighbour
    const float away = __int_as_float(__float_as_int(ac) + 1), toward = __int_as_float(__float_as_int(ac) - 1);
    const float half = ((d >= 0.0f) == (c >= 0.0f)) ? 0.5f * (away - ac) : 0.5f * (ac - toward);
    if (fabsf(d) + ac * 0x1p-40f < half) return c;
    return __double2float_rn(__dmul_rn(__ddiv_rn(__dsub_rn((double)S, 1.0), (double)lam), (double)k));
}

struct PbdConst {
    float stretch[3], shear[3], eps;
};

// solveStrainConstraints (PosBaseDynamic.cpp:55-117) for one tet: p[c].xyz
// the corner positions, p[c].w the inverse masses, D = Dm^-1 row-major.
__device__ __forceinline__ void pbd_project(const float4 p[4], const float D[9], const PbdConst &k, float dp[4][3]) {
    const float pw[4] = {p[0].w, p[1].w, p[2].w, p[3].w};
#pragma unroll
    for (int c = 0; c < 4; ++c) dp[c][0] = dp[c][1] = dp[c][2] = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            const float x0[3] = {fadd(p[0].x, dp[0][0]), fadd(p[0].y, dp[0][1]), fadd(p[0].z, dp[0][2])};
            float P[3][3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float4 &q = p[c + 1];
                P[0][c] = fsub(fadd(q.x, dp[c + 1][0]), x0[0]);
                P[1][c] = fsub(fadd(q.y, dp[c + 1][1]), x0[1]);
                P[2][c] = fsub(fadd(q.z, dp[c + 1][2]), x0[2]);
            }
            float fi[3], fj[3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                fi[r] = fadd(fadd(fmul(P[r][0], D[i]), fmul(P[r][1], D[3 + i])), fmul(P[r][2], D[6 + i]));
                fj[r] = fadd(fadd(fmul(P[r][0], D[j]), fmul(P[r][1], D[3 + j])), fmul(P[r][2], D[6 + j]));
            }
            const float S = dot3e(fi, fj);
            float d[4][3];
#pragma unroll
            for (int r = 0; r < 3; ++r) d[0][r] = 0.f;
#pragma unroll
            for (int kk = 0; kk < 3; ++kk)
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    d[kk + 1][r] = fadd(fmul(fj[r], D[3 * kk + i]), fmul(fi[r], D[3 * kk + j]));
                    d[0][r] = fsub(d[0][r], d[kk + 1][r]);
                }
            float lam = fmul(pw[0], dot3e(d[0], d[0]));
            lam = fadd(lam, fmul(pw[1], dot3e(d[1], d[1])));
            lam = fadd(lam, fmul(pw[2], dot3e(d[2], d[2])));
            lam = fadd(lam, fmul(pw[3], dot3e(d[3], d[3])));
            if (lam < k.eps) continue;
            if (i == j) lam = pbd_stretch_mult(S, lam, k.stretch[i]);
            else lam = fmul(__fdiv_rn(S, lam), k.shear[i + j - 1]);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float s = fmul(lam, pw[c]);
#pragma unroll
                for (int r = 0; r < 3; ++r) dp[c][r] = fsub(dp[c][r], fmul(s, d[c][r]));
            }
        }
    }
}

// A level-ordered tet's static record (ids, Dm^-1 rows).
struct PbdTet {
    int4 q;
    float4 r0, r1, r2;
};

__device__ __forceinline__ PbdTet pbd_load(const PbdView &v, int j) {
    PbdTet t;
    t.q = __ldg(v.tet + j);
    t.r0 = __ldg(v.d0 + j);
    t.r1 = __ldg(v.d1 + j);
    t.r2 = __ldg(v.d2 + j);
    return t;
}

__device__ __forceinline__ void pbd_apply(const PbdView &v, const PbdTet &t, const PbdConst &k) {
    const float D[9] = {t.r0.x, t.r0.y, t.r0.z, t.r1.x, t.r1.y, t.r1.z, t.r2.x, t.r2.y, t.r2.z};
    const int id[4] = {t.q.x, t.q.y, t.q.z, t.q.w};
    float4 p[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) p[c] = __ldcg(v.px + id[c]);
    float dp[4][3];
    pbd_project(p, D, k, dp);
#pragma unroll
    for (int c = 0; c < 4; ++c)
        v.px[id[c]] = make_float4(fadd(p[c].x, dp[c][0]), fadd(p[c].y, dp[c][1]), fadd(p[c].z, dp[c][2]), p[c].w);
}

// The sweeps' schedule.  Sweep q runs level l of its group at step l + q D: with
// D larger than any level difference between tets that share a node (the
// group's delay), a tet comes after every earlier tet of its own sweep that
// shares a node (their levels are lower), after all such tets of the sweep
// before (their levels are at most its own + D - 1, D steps earlier) and before
// those of the next one, so it reads what the serial order gives it; and tets
// of one step share no node.  L + (sweeps - 1) D steps instead of L sweeps:
// the dependent chain of a level, which bounds a step, then serves several
// sweeps at once.  On structured meshes D is 2-10% of L (the 1M-tet box: L
// 2,325, D 39; the 24,000-tet bar 348 and 34), on meshes in arbitrary order up
// to L, where the sweeps simply follow one another.
struct PbdStep {
    int l0, L, D, sweeps, steps;
    __device__ PbdStep(const PbdView &v, int g, int iterations) {
        l0 = v.grp[g];
        L = v.grp[g + 1] - l0;
        D = v.delay[g];
        sweeps = iterations;
        steps = L > 0 && iterations > 0 ? L + (iterations - 1) * D : 0;
    }
    // the sweeps that are on at step t: q0 .. q1
    __device__ __forceinline__ void on(int t, int &q0, int &q1) const {
        q0 = t < L ? 0 : (t - L) / D + 1;
        q1 = min(sweeps - 1, t / D);
    }
    // CTA `rank`'s run of the level of sweep q at step t: its first tet, count
    __device__ __forceinline__ void run(const PbdView &v, int t, int q, int rank, int csize, int &b0, int &n) const {
        const int l = l0 + t - q * D;
        const int a = __ldg(v.lvl + l), e = __ldg(v.lvl + l + 1);
        const int chunk = (e - a + csize - 1) / csize;
        b0 = a + rank * chunk;
        n = max(0, min(chunk, e - b0));
    }
    // the tet at place `pos` of CTA `rank`'s runs of step t, -1 past their end
    __device__ __forceinline__ int tet(const PbdView &v, int t, int rank, int csize, int pos) const {
        int q0, q1;
        on(t, q0, q1);
        for (int q = q0; q <= q1; ++q) {
            int b0, n;
            run(v, t, q, rank, csize, b0, n);
            if (pos < n) return b0 + pos;
            pos -= n;
        }
        return -1;
    }
};

// Scheduler warp: the first kPbdWorkers tets of CTA `rank`'s runs of step t
// into idx (-1 past their end).
__device__ __forceinline__ void pbd_schedule(const PbdStep &sch, const PbdView &v, int t, int rank, int csize, int *idx) {
    const int lane = threadIdx.x & 31;
    int q0, q1, base = 0;
    sch.on(t, q0, q1);
    for (int qa = q0; qa <= q1 && base < kPbdWorkers; qa += 32) {
        int b0 = 0, n = 0;
        if (qa + lane <= q1) sch.run(v, t, qa + lane, rank, csize, b0, n);
        int end = n;  // inclusive prefix sum over the lanes
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += x;
        }
        const int cnt = min(32, q1 - qa + 1);
        for (int i = 0; i < cnt; ++i) {
            const int ni = __shfl_sync(0xffffffffu, n, i), bi = __shfl_sync(0xffffffffu, b0, i);
            const int at = base + __shfl_sync(0xffffffffu, end, i) - ni;
            for (int x = lane; x < ni && at + x < kPbdWorkers; x += 32) idx[at + x] = bi + x;
        }
        base += __shfl_sync(0xffffffffu, end, 31);
    }
    for (int x = base + lane; x < kPbdWorkers; x += 32) idx[x] = -1;
}

// One cluster per group of levels (an instance); a step's tets are split into
// one contiguous run per level and CTA of the cluster.  The cluster barrier
// orders one step's position writes before the next one's reads.  A scheduler
// warp beside the workers lists the CTA's tets of the step after next, so that
// a worker loads the next step's static record before this step's chain and
// a step is that chain alone: position loads, the projections, the barrier.
// (Looked up by every worker between the barrier's arrive and wait, five
// sweeps of the 1M-tet box took 13.2 instead of 10.2 ms, of the 24,000-tet
// bar 2.31 instead of 1.28.)
template <class Load, class Apply>
__device__ __forceinline__ void pbd_run(cg::cluster_group &cl, const PbdView &v, int g, int iterations, Load load,
                                        Apply apply) {
    __shared__ int s_idx[2][kPbdWorkers];
    const int csize = (int)cl.num_blocks(), rank = (int)cl.block_rank(), tid = (int)threadIdx.x;
    const PbdStep sch(v, g, iterations);
    const bool worker = tid < kPbdWorkers;
    if (sch.steps == 0) return;  // uniform over the cluster
    if (!worker) {
        pbd_schedule(sch, v, 0, rank, csize, s_idx[0]);
        if (sch.steps > 1) pbd_schedule(sch, v, 1, rank, csize, s_idx[1]);
    }
    __syncthreads();
    int j = worker ? s_idx[0][tid] : -1;
    bool full = s_idx[0][kPbdWorkers - 1] >= 0;  // the step may have more tets than workers
    PbdTet cur;
    if (j >= 0) cur = load(j);
    __syncthreads();
    for (int t = 0; t < sch.steps; ++t) {
        if (worker) {
            const int jn = t + 1 < sch.steps ? s_idx[(t + 1) & 1][tid] : -1;
            const bool fulln = t + 1 < sch.steps && s_idx[(t + 1) & 1][kPbdWorkers - 1] >= 0;
            PbdTet nxt = cur;
            if (jn >= 0) nxt = load(jn);
            if (j >= 0) {
                apply(cur);
                // (levels wider than the cluster's workers)
                if (full)
                    for (int pos = tid + kPbdWorkers, x; (x = sch.tet(v, t, rank, csize, pos)) >= 0; pos += kPbdWorkers)
                        apply(load(x));
            }
            cur = nxt;
            j = jn;
            full = fulln;
        } else if (t + 2 < sch.steps) {
            pbd_schedule(sch, v, t + 2, rank, csize, s_idx[t & 1]);
        }
        cl.sync();
    }
}

// Positions in global memory, read through L2 (ld.global.cg).
__global__ void __launch_bounds__(kPbdThreads) k_pbd_sweep(PbdView v, int iterations, PbdConst k) {
    cg::cluster_group cl = cg::this_cluster();
    const int g = blockIdx.x / (int)cl.num_blocks();
    pbd_run(cl, v, g, iterations, [&](int j) { return pbd_load(v, j); }, [&](const PbdTet &t) { pbd_apply(v, t, k); });
}

// The same sweep with the instance's positions held in the cluster's
// distributed shared memory: CTA r of the 16 keeps nodes r, r + 16, ... of the
// instance, and a tet corner is addressed by its code (owner CTA << 16 |
// offset), so every step's position loads and stores go SM to SM instead of
// through L2, and the cluster barrier releases shared-memory writes only.
// Interleaved, because a level's tets lie near one another: with contiguous
// slices one or two CTAs served a level's whole traffic (10.3 instead of 8.7
// ms for five sweeps of the 1M-tet box).
// Used when an instance's nodes fit (S * 16 B of dynamic shared memory a CTA).
__device__ __forceinline__ float4 *dsm_node(cg::cluster_group &cl, float4 *s_px, int code) {
    return cl.map_shared_rank(s_px, (unsigned)code >> 16) + (code & 0xffff);
}

__global__ void __launch_bounds__(kPbdThreads)
    k_pbd_sweep_dsmem(PbdView v, const int4 *codes, const int4 *gnode, int iterations, PbdConst k) {
    extern __shared__ float4 s_px[];
    cg::cluster_group cl = cg::this_cluster();
    const int g = blockIdx.x / (int)cl.num_blocks();
    const int rank = (int)cl.block_rank();
    const int4 gn = gnode[g];  // {first padded node, slice S, node count}
    const int nb = gn.x, S = gn.y, cnt = gn.z;
    for (int j = threadIdx.x; j < S; j += blockDim.x) {
        const int n = j * kPbdClusterMax + rank;
        if (n < cnt) s_px[j] = v.px[nb + n];
    }
    cl.sync();
    PbdView vc = v;  // the static records with corner codes in place of node ids
    vc.tet = codes;
    pbd_run(
        cl, vc, g, iterations, [&](int j) { return pbd_load(vc, j); },
        [&](const PbdTet &t) {
            const float D[9] = {t.r0.x, t.r0.y, t.r0.z, t.r1.x, t.r1.y, t.r1.z, t.r2.x, t.r2.y, t.r2.z};
            float4 *ptr[4] = {dsm_node(cl, s_px, t.q.x), dsm_node(cl, s_px, t.q.y), dsm_node(cl, s_px, t.q.z),
                              dsm_node(cl, s_px, t.q.w)};
            float4 p[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) p[c] = *ptr[c];
            float dp[4][3];
            pbd_project(p, D, k, dp);
#pragma unroll
            for (int c = 0; c < 4; ++c)
                *ptr[c] = make_float4(fadd(p[c].x, dp[c][0]), fadd(p[c].y, dp[c][1]), fadd(p[c].z, dp[c][2]), p[c].w);
        });
    // (the last barrier ordered every position before the copy out)
    for (int j = threadIdx.x; j < S; j += blockDim.x) {
        const int n = j * kPbdClusterMax + rank;
        if (n < cnt) v.px[nb + n] = s_px[j];
    }
}

// slot of column `target` in block row [b, e) (columns ascending), e if absent
__device__ __forceinline__ int col_slot(const int *col, int b, int e, int target) {
    int lo = b, hi = e;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (col[mid] < target) lo = mid + 1;
        else hi = mid;
    }
    return (lo < e && col[lo] == target) ? lo : e;
}

// 1 / lumped mass as the reference forms it (1.0 / m: an FP64 quotient
// rounded to FP32, TetMesh.cpp:209), 0 at a pinned node
__device__ __forceinline__ float inv_mass_of(const float4 &info) {
    return info.z == 1.f ? 0.f : __double2float_rn(__ddiv_rn(1.0, (double)info.x));
}

__device__ __forceinline__ float4 state_pos4(const DevMesh &m, const DevState &st, int i) {
    const float4 X = m.rest[i], h = st.u0h[i], l = st.u0l[i];
    return make_float4(state_position(X.x, h.x, l.x), state_position(X.y, h.y, l.y), state_position(X.z, h.z, l.z),
                       0.f);
}

// f = gravity + ext of a node (the caller's forces; the pin spring that
// TetMesh::computeExternalForces puts on a pinned node is multiplied by its
// zero inverse mass in both integrators)
__device__ __forceinline__ float3 node_force(const float4 &info, const float4 *ext, int i) {
    float3 f = make_float3(0.f, info.y, 0.f);
    if (ext) {
        const float4 e = ext[i];
        f = make_float3(fadd(f.x, e.x), fadd(f.y, e.y), fadd(f.z, e.z));
    }
    return f;
}

// ---- the PBD step's rest data, formed exactly as TetMesh::initModel does in
// FP32 (TetMesh.cpp:186-216) with Eigen 3.2's 3x3 determinant (row-0
// cofactor expansion) and inverse (adjugate of the column-0 cofactors times
// 1 / det): the sweeps then see the reference's own Dm^-1 and masses.
__device__ __forceinline__ float eig_cof(const float m[3][3], int i, int j) {
    const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
    return fsub(fmul(m[i1][j1], m[i2][j2]), fmul(m[i1][j2], m[i2][j1]));
}

// level-ordered tet j (padded tet order[j]): Dm^-1 rows, and its lumped-mass
// share vol / 4 * density by padded tet
__global__ void k_pbd_rest(DevMesh m, const int *order, int n, float density, float4 *d0, float4 *d1, float4 *d2,
                           float *share) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int tp = order[j];
    const int4 q = m.tets[tp];
    const float4 X0 = m.rest[q.x], X1 = m.rest[q.y], X2 = m.rest[q.z], X3 = m.rest[q.w];
    const float m_[3][3] = {{fsub(X1.x, X0.x), fsub(X2.x, X0.x), fsub(X3.x, X0.x)},
                            {fsub(X1.y, X0.y), fsub(X2.y, X0.y), fsub(X3.y, X0.y)},
                            {fsub(X1.z, X0.z), fsub(X2.z, X0.z), fsub(X3.z, X0.z)}};
    const float det = fadd(fsub(fmul(m_[0][0], fsub(fmul(m_[1][1], m_[2][2]), fmul(m_[1][2], m_[2][1]))),
                                fmul(m_[0][1], fsub(fmul(m_[1][0], m_[2][2]), fmul(m_[1][2], m_[2][0])))),
                           fmul(m_[0][2], fsub(fmul(m_[1][0], m_[2][1]), fmul(m_[1][1], m_[2][0]))));
    const float vol = __double2float_rn(__ddiv_rn((double)fabsf(det), 6.0));
    share[tp] = __double2float_rn(__dmul_rn(__ddiv_rn((double)vol, 4.0), (double)density));
    const float c0[3] = {eig_cof(m_, 0, 0), eig_cof(m_, 1, 0), eig_cof(m_, 2, 0)};
    const float d = fadd(fmul(c0[0], m_[0][0]), fadd(fmul(c0[1], m_[1][0]), fmul(c0[2], m_[2][0])));
    const float inv = __fdiv_rn(1.0f, d);
    d0[j] = make_float4(fmul(c0[0], inv), fmul(c0[1], inv), fmul(c0[2], inv), 0.f);
    d1[j] = make_float4(fmul(eig_cof(m_, 0, 1), inv), fmul(eig_cof(m_, 1, 1), inv), fmul(eig_cof(m_, 2, 1), inv), 0.f);
    d2[j] = make_float4(fmul(eig_cof(m_, 0, 2), inv), fmul(eig_cof(m_, 1, 2), inv), fmul(eig_cof(m_, 2, 2), inv), 0.f);
}

// per node: lumped mass summed in tet order, {1 / mass (FP64 quotient
// rounded; 0 when pinned), -gravity * mass}
__global__ void k_pbd_mass(DevMesh m, const float *share, float gravity, float2 *node) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.Np) return;
    const float4 info = m.info[i];
    if (info.z == 2.f) { node[i] = make_float2(0.f, 0.f); return; }
    float s = 0.f;
    for (int j = m.inc_ptr[i]; j < m.inc_ptr[i + 1]; ++j) s = fadd(s, share[m.inc[j] >> 2]);
    node[i] = make_float2(info.z == 1.f ? 0.f : __double2float_rn(__ddiv_rn(1.0, (double)s)), fmul(-gravity, s));
}

// p = x + dt (v + (dt w) f), px = (p, w), x0 = x (PosBaseDynamic.cpp:24-30);
// node = {w, gravity_y} of the PBD rest data
__global__ void k_pbd_begin(DevMesh m, DevState st, const float2 *node, const float4 *ext, float dt, float4 *px,
                            float4 *x0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.Np) return;
    const float4 info = m.info[i];
    if (info.z == 2.f) { px[i] = x0[i] = make_float4(0.f, 0.f, 0.f, 0.f); return; }
    const float4 x = state_pos4(m, st, i), v = st.v[i];
    const float2 nd = node[i];
    const float w = nd.x, s = fmul(dt, w);
    float3 f = make_float3(0.f, nd.y, 0.f);
    if (ext) {
        const float4 e = ext[i];
        f = make_float3(fadd(f.x, e.x), fadd(f.y, e.y), fadd(f.z, e.z));
    }
    px[i] = make_float4(fadd(x.x, fmul(dt, fadd(v.x, fmul(s, f.x)))), fadd(x.y, fmul(dt, fadd(v.y, fmul(s, f.y)))),
                        fadd(x.z, fmul(dt, fadd(v.z, fmul(s, f.z)))), w);
    x0[i] = x;
}

// x = p and v = ((p - x) 0.99) / dt (PosBaseDynamic.cpp:51-52), or, with
// divide_first, ((p - x) / dt) 0.99 (ProjDynamic.cpp:477-478); the state keeps
// p - X exactly as (hi, lo)
__global__ void k_dyn_end(DevMesh m, DevState st, const float4 *px, const float4 *x0, float dt, int divide_first) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.Np || m.info[i].z == 2.f) return;
    const float4 p = px[i], x = x0[i], X = m.rest[i];
    const float c = 0.99f;
    float3 v;
    if (divide_first)
        v = make_float3(fmul(__fdiv_rn(fsub(p.x, x.x), dt), c), fmul(__fdiv_rn(fsub(p.y, x.y), dt), c),
                        fmul(__fdiv_rn(fsub(p.z, x.z), dt), c));
    else
        v = make_float3(__fdiv_rn(fmul(fsub(p.x, x.x), c), dt), __fdiv_rn(fmul(fsub(p.y, x.y), c), dt),
                        __fdiv_rn(fmul(fsub(p.z, x.z), c), dt));
    float h[3], l[3];
    two_sum(p.x, -X.x, h[0], l[0]);
    two_sum(p.y, -X.y, h[1], l[1]);
    two_sum(p.z, -X.z, h[2], l[2]);
    st.u0h[i] = make_float4(h[0], h[1], h[2], 0.f);
    st.u0l[i] = make_float4(l[0], l[1], l[2], 0.f);
    st.v[i] = make_float4(v.x, v.y, v.z, 0.f);
}

// ---------------------------------------------------------------- projective dynamics
// Row i of A = M / dt_m^2 + sum_t k vol_t (w_a . w_b) I3, one value a block
// (A.scalar), in the node's incidence order; D^-1 = 1 / a_ii.
__global__ void __launch_bounds__(128) k_pd_assemble(DevMesh m, BsrView A, float inv_dt2, float stiffness,
                                                     float *dinv9) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.Np) return;
    const int rb = A.ptr[i], re = A.ptr[i + 1];
    float *row = A.val + rb;
    for (int k = 0; k < re - rb; ++k) row[k] = 0.f;
    const float4 info = m.info[i];
    if (info.z != 2.f) {
        for (int j = m.inc_ptr[i]; j < m.inc_ptr[i + 1]; ++j) {
            const int ent = m.inc[j], t = ent >> 2, c = ent & 3;
            const int4 q = m.tets[t];
            const int qn[4] = {q.x, q.y, q.z, q.w};
            const float4 r0 = m.row0[t], r1 = m.row1[t], r2 = m.row2[t];
            const float w[4][3] = {{-(r0.x + r1.x + r2.x), -(r0.y + r1.y + r2.y), -(r0.z + r1.z + r2.z)},
                                   {r0.x, r0.y, r0.z},
                                   {r1.x, r1.y, r1.z},
                                   {r2.x, r2.y, r2.z}};
            const float kv = stiffness * fabsf(r0.w);
            for (int cc = 0; cc < 4; ++cc) {
                const int sl = col_slot(A.col, rb, re, qn[cc]);
                if (sl == re) continue;  // (the pattern holds every tet's node pairs)
                row[sl - rb] += kv * (w[c][0] * w[cc][0] + w[c][1] * w[cc][1] + w[c][2] * w[cc][2]);
            }
        }
    }
    const int dsl = col_slot(A.col, rb, re, i);
    float inv = 0.f;
    if (dsl < re) {
        row[dsl - rb] += info.z == 2.f ? 1.f : info.x * inv_dt2;
        inv = 1.f / row[dsl - rb];
    }
    for (int k = 0; k < 9; ++k) dinv9[9 * (size_t)i + k] = (k % 4 == 0) ? inv : 0.f;
}

// q = dt v + (dt^2 w) f, the inertial target's offset from x (the reference's
// s = (x + dt v + dt^2 w f) m / dt^2, ProjDynamic.cpp:447-463, is
// m / dt^2 (x + q)); p = x0 = x
__global__ void k_pd_begin(DevMesh m, DevState st, const float4 *ext, float dt, float4 *q, float4 *px, float4 *x0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.Np) return;
    const float4 info = m.info[i];
    if (info.z == 2.f) {
        q[i] = px[i] = x0[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const float4 x = state_pos4(m, st, i), v = st.v[i];
    const float dt2 = fmul(dt, dt), a = fmul(dt2, inv_mass_of(info));
    const float3 f = node_force(info, ext, i);
    q[i] = make_float4(fadd(fmul(dt, v.x), fmul(a, f.x)), fadd(fmul(dt, v.y), fmul(a, f.y)),
                       fadd(fmul(dt, v.z), fmul(a, f.z)), 0.f);
    px[i] = x;
    x0[i] = x;
}

// Per tet: R = U V^T with JacobiSVD's determinant fix (first, largest
// columns negated), i.e. U diag(sg, 1, sg) V^T of the modified SVD
// (sg = sign of the smallest singular value).  Corner a's share of the
// global step's residual, k vol (R - F) w_a (its projection k vol R w_a
// less its share of A p, both from edge differences: no absolute coordinate
// enters), goes into its gather slot.
__global__ void __launch_bounds__(128) k_pd_local(DevMesh m, const float4 *px, float stiffness, float4 *slot) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m.Tp) return;
    const int4 q = m.tets[t];
    if (q.x < 0) return;
    const float4 r0 = m.row0[t], r1 = m.row1[t], r2 = m.row2[t];
    const float dinv[9] = {r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r2.x, r2.y, r2.z};
    const float4 x0 = px[q.x], x1 = px[q.y], x2 = px[q.z], x3 = px[q.w];
    const float ds[3][3] = {{x1.x - x0.x, x2.x - x0.x, x3.x - x0.x},
                            {x1.y - x0.y, x2.y - x0.y, x3.y - x0.y},
                            {x1.z - x0.z, x2.z - x0.z, x3.z - x0.z}};
    float G[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            G[3 * r + c] = ds[r][0] * dinv[c] + ds[r][1] * dinv[3 + c] + ds[r][2] * dinv[6 + c] - (r == c ? 1.f : 0.f);
    float U[9], sv[3], V[9], sign3;
    svd_disp<float, 4>(G, U, sv, V, sign3);
    const float sg = sign3 < 0.f ? -1.f : 1.f;
    float E[9];  // R - F = R - I - G
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            E[3 * r + c] = (sg * U[3 * r] * V[3 * c] + U[3 * r + 1] * V[3 * c + 1] + sg * U[3 * r + 2] * V[3 * c + 2] -
                            (r == c ? 1.f : 0.f)) - G[3 * r + c];
    const float kv = stiffness * fabsf(r0.w);
    const float w[4][3] = {{-(r0.x + r1.x + r2.x), -(r0.y + r1.y + r2.y), -(r0.z + r1.z + r2.z)},
                           {r0.x, r0.y, r0.z},
                           {r1.x, r1.y, r1.z},
                           {r2.x, r2.y, r2.z}};
    const int4 sl = m.tslot[t];
    const int sls[4] = {sl.x, sl.y, sl.z, sl.w};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        slot[sls[a]] = make_float4(kv * (E[0] * w[a][0] + E[1] * w[a][1] + E[2] * w[a][2]),
                                   kv * (E[3] * w[a][0] + E[4] * w[a][1] + E[5] * w[a][2]),
                                   kv * (E[6] * w[a][0] + E[7] * w[a][1] + E[8] * w[a][2]), 0.f);
    }
}

// The global step's residual r = b - A p = m / dt_m^2 (x - p) + m / dt^2 q
// + (m / dt^2 - m / dt_m^2) x (zero unless A was formed with another time
// step) + the node's (R - F) slots in incidence order (ascending tet, as the
// reference's m_proj_idx lists them); the correction d = 0
__global__ void k_pd_rhs(DevMesh m, const float4 *q, const float4 *x0, const float4 *px, const float4 *slot,
                         float inv_dt2, float inv_dtm2, float4 *r, float4 *d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.Np) return;
    d[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 info = m.info[i];
    if (info.z == 2.f) { r[i] = d[i]; return; }
    const float4 qq = q[i], x = x0[i], p = px[i];
    const float mb = info.x * inv_dt2, mm = info.x * inv_dtm2, mx = mb - mm;
    float4 a = make_float4(mm * (x.x - p.x) + mb * qq.x, mm * (x.y - p.y) + mb * qq.y, mm * (x.z - p.z) + mb * qq.z, 0.f);
    if (mx != 0.f) {
        a.x += mx * x.x;
        a.y += mx * x.y;
        a.z += mx * x.z;
    }
    for (int j = m.inc_ptr[i]; j < m.inc_ptr[i + 1]; ++j) {
        const float4 c = slot[j];
        a.x += c.x;
        a.y += c.y;
        a.z += c.z;
    }
    r[i] = a;
}

__global__ void k_pd_apply(int Np, float4 *p, const float4 *d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Np) return;
    const float4 a = p[i], c = d[i];
    p[i] = make_float4(a.x + c.x, a.y + c.y, a.z + c.z, a.w);
}

}  // namespace

cudaError_t launch_pd_apply(cudaStream_t s, int Np, float4 *p, const float4 *d) {
    k_pd_apply<<<(Np + 255) / 256, 256, 0, s>>>(Np, p, d);
    return cudaGetLastError();
}

cudaError_t launch_pbd_rest(cudaStream_t s, const DevMesh &m, const int *order, int n, float density, float gravity,
                            float4 *d0, float4 *d1, float4 *d2, float *share, float2 *node) {
    if (n > 0) k_pbd_rest<<<(n + 127) / 128, 128, 0, s>>>(m, order, n, density, d0, d1, d2, share);
    k_pbd_mass<<<(m.Np + 255) / 256, 256, 0, s>>>(m, share, gravity, node);
    return cudaGetLastError();
}

cudaError_t launch_pbd_begin(cudaStream_t s, const DevMesh &m, const DevState &st, const float2 *node,
                             const float4 *ext, float dt, float4 *px, float4 *x0) {
    k_pbd_begin<<<(m.Np + 255) / 256, 256, 0, s>>>(m, st, node, ext, dt, px, x0);
    return cudaGetLastError();
}

cudaError_t launch_pbd_sweeps(cudaStream_t s, const PbdView &v, int n_groups, int iterations, const float stretch[3],
                              const float shear[3]) {
    PbdConst k;
    for (int i = 0; i < 3; ++i) { k.stretch[i] = stretch[i]; k.shear[i] = shear[i]; }
    k.eps = 1e-6f;
    static int big_ok = -1;  // whether 16-CTA clusters of this kernel can be resident
    if (big_ok < 0) {
        big_ok = 0;
        if (cudaFuncSetAttribute(k_pbd_sweep, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            cudaLaunchConfig_t q = {};
            q.gridDim = dim3(kPbdClusterMax);
            q.blockDim = dim3(kPbdThreads);
            cudaLaunchAttribute qa;
            qa.id = cudaLaunchAttributeClusterDimension;
            qa.val.clusterDim.x = kPbdClusterMax;
            qa.val.clusterDim.y = 1;
            qa.val.clusterDim.z = 1;
            q.attrs = &qa;
            q.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, k_pbd_sweep, &q) == cudaSuccess && n > 0) big_ok = 1;
        }
        cudaGetLastError();  // a refused query leaves no error behind
    }
    const int csize = (big_ok && n_groups <= 4) ? kPbdClusterMax : 8;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_groups * csize);
    cfg.blockDim = dim3(kPbdThreads);
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = csize;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_pbd_sweep, v, iterations, k);
}

bool pbd_dsmem_fits(int smem_bytes) {
    if (smem_bytes > 227 * 1024) return false;
    if (cudaFuncSetAttribute(k_pbd_sweep_dsmem, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        allow_all_smem(k_pbd_sweep_dsmem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t q = {};
    q.gridDim = dim3(kPbdClusterMax);
    q.blockDim = dim3(kPbdThreads);
    q.dynamicSmemBytes = smem_bytes;
    cudaLaunchAttribute qa;
    qa.id = cudaLaunchAttributeClusterDimension;
    qa.val.clusterDim.x = kPbdClusterMax;
    qa.val.clusterDim.y = 1;
    qa.val.clusterDim.z = 1;
    q.attrs = &qa;
    q.numAttrs = 1;
    int n = 0;
    const bool ok = cudaOccupancyMaxActiveClusters(&n, k_pbd_sweep_dsmem, &q) == cudaSuccess && n > 0;
    cudaGetLastError();
    return ok;
}

cudaError_t launch_pbd_sweeps_dsmem(cudaStream_t s, const PbdView &v, const int4 *codes, const int4 *gnode,
                                    int n_groups, int smem_bytes, int iterations, const float stretch[3],
                                    const float shear[3]) {
    PbdConst k;
    for (int i = 0; i < 3; ++i) { k.stretch[i] = stretch[i]; k.shear[i] = shear[i]; }
    k.eps = 1e-6f;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_groups * kPbdClusterMax);
    cfg.blockDim = dim3(kPbdThreads);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kPbdClusterMax;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_pbd_sweep_dsmem, v, codes, gnode, iterations, k);
}

cudaError_t launch_dyn_end(cudaStream_t s, const DevMesh &m, const DevState &st, const float4 *px, const float4 *x0,
                           float dt, int divide_first) {
    k_dyn_end<<<(m.Np + 255) / 256, 256, 0, s>>>(m, st, px, x0, dt, divide_first);
    return cudaGetLastError();
}

cudaError_t launch_pd_assemble(cudaStream_t s, const DevMesh &m, const BsrView &A, float dt_matrix, float stiffness,
                               float *dinv9) {
    k_pd_assemble<<<(m.Np + 127) / 128, 128, 0, s>>>(m, A, 1.f / (dt_matrix * dt_matrix), stiffness, dinv9);
    return cudaGetLastError();
}

cudaError_t launch_pd_begin(cudaStream_t s, const DevMesh &m, const DevState &st, const float4 *ext, float dt,
                            float4 *q, float4 *px, float4 *x0) {
    k_pd_begin<<<(m.Np + 255) / 256, 256, 0, s>>>(m, st, ext, dt, q, px, x0);
    return cudaGetLastError();
}

cudaError_t launch_pd_residual(cudaStream_t s, const DevMesh &m, const float4 *px, float stiffness, float dt,
                               float dt_matrix, float4 *slot, const float4 *q, const float4 *x0, float4 *r, float4 *d) {
    k_pd_local<<<(m.Tp + 127) / 128, 128, 0, s>>>(m, px, stiffness, slot);
    k_pd_rhs<<<(m.Np + 255) / 256, 256, 0, s>>>(m, q, x0, px, slot, 1.f / (dt * dt),
                                                1.f / (dt_matrix * dt_matrix), r, d);
    return cudaGetLastError();
}

}  // namespace pbs

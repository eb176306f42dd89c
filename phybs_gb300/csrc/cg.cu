// Block-Jacobi preconditioned conjugate gradients on the node matrix of the
// backward-Euler and projective-dynamics steps, one cooperative launch a solve.
//
// A solve of hundreds of iterations as five kernels an iteration was bound by
// its launches on small meshes (20 us an iteration at 5,000 rows) and by
// uncoalesced matrix rows and FP64 dot products on large ones (36 us at
// 210,000 rows with one value a block).  This takes 6.7 us and 15 us.  What
// bounds it now: the two sums, 2-3 us each from their lane trees and the
// words' round trip, and at 210,000 rows the shared-memory reads of the
// direction vector (4.2 us).  Here every CTA (one a SM) owns a run
// of rows of the Morton order for the whole solve and keeps what fits in
// shared memory: the direction vector of its rows and of the neighbours they
// multiply (the halo), its residual, q and x, and its share of the matrix.
// An iteration exchanges words through L2 (exchange.cuh):
//   p     each row's direction, read by the CTAs whose halo it is in;
//   p.q   and  r.z (r.r)   one word a sum and CTA, {hi, lo, check, tag}, read
//         by every CTA, which adds them in the same order and so takes the
//         same decisions.
// A direction word is overwritten after a sum that its readers contribute to
// once they have read it.  The words of two sums in a row alternate between
// two buffers: a CTA writes a buffer again after the sum between, which every
// CTA contributes to once it has read the buffer.
//
// The matrix is kept in slices of 32 rows, entry by entry (sliced ELLPACK), so
// a warp's loads of one entry are contiguous, with 16-bit columns into the
// CTA's direction vector.  Rows of a CTA are ordered by length, so a slice's
// rows end together, and the words of p are kept by row place, so that writing
// and gathering them is contiguous (by node id the exchange took 11,700 cycles
// of an iteration instead of 3,900 at 210,000 rows).
//
// Dot products run in double-float on vectors scaled by powers of two (GB300's
// FP64 pipe took longer for them than memory for the matrix): products exact,
// sums to about 2^-44.  With FP64 sums the outputs' errors against 64 bits were
// the same to four digits on twenty systems of 300 to 37,000 rows.  The scales bring the largest |b| and |D^-1 b| to [1, 2),
// so that no square leaves FP32's range.
#include <climits>

#include <cuda_runtime.h>

#include "../../include/phybs.h"
#include "exchange.cuh"
#include "phybs_internal.cuh"
#include "tet_math.cuh"

namespace pbs {

namespace {

__device__ __forceinline__ float4 f4(float x, float y, float z) { return make_float4(x, y, z, 0.f); }

// ------------------------------------------------------------ pattern
// Row i's columns: itself and every node it shares a tet with, ascending.
// Selected one after the other as the smallest beyond the last, without scratch:
// quadratic in the incident tets, so the rows of nodes with more than
// BSR_HUB_TETS of them are left to the host, which sorts (a node of 12,000 tets
// would take one thread seconds).
__device__ __forceinline__ int next_col(const DevMesh &m, int i, int last) {
    int best = i > last ? i : INT_MAX;
    for (int j = m.inc_ptr[i]; j < m.inc_ptr[i + 1]; ++j) {
        const int4 q = m.tets[m.inc[j] >> 2];
        if (q.x > last) best = min(best, q.x);
        if (q.y > last) best = min(best, q.y);
        if (q.z > last) best = min(best, q.z);
        if (q.w > last) best = min(best, q.w);
    }
    return best;
}

__global__ void k_bsr_count(DevMesh m, int *cnt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.Np) return;
    int n = 0;
    if (m.inc_ptr[i + 1] - m.inc_ptr[i] > BSR_HUB_TETS) n = -1;
    else
        for (int c = next_col(m, i, -1); c != INT_MAX; c = next_col(m, i, c)) ++n;
    cnt[i] = n;
}

__global__ void k_bsr_fill(DevMesh m, const int *ptr, int *col) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.Np) return;
    if (m.inc_ptr[i + 1] - m.inc_ptr[i] > BSR_HUB_TETS) return;
    int k = ptr[i];
    for (int c = next_col(m, i, -1); c != INT_MAX; c = next_col(m, i, c)) col[k++] = c;
}

// ------------------------------------------------------------ sliced values
// Values of the rows and their block-Jacobi inverses in slice order.  NV = 9:
// the nine entries of a block as nine planes of 32 lanes.
template <int NV> __global__ void k_cg_pack(CgPlanView pl, BsrView A, const float *dinv9, float *out, float *dinv) {
    const int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (s >= pl.n_slices) return;
    const int i = pl.srow[32 * (size_t)s + lane];
    if (i < 0) return;
#pragma unroll
    for (int c = 0; c < NV; ++c) dinv[(size_t)s * (32 * NV) + c * 32 + lane] = dinv9[9 * (size_t)i + c];
    const int rb = A.ptr[i], n = A.ptr[i + 1] - rb;
    const size_t off = (size_t)pl.soff[s];
    for (int k = 0; k < n; ++k)
#pragma unroll
        for (int c = 0; c < NV; ++c) out[(off + k) * (32 * NV) + c * 32 + lane] = A.val[(size_t)(rb + k) * NV + c];
}

// ------------------------------------------------------------ the solve
// a . b of vectors scaled by powers of two, in double-float.
__device__ __forceinline__ DFloat dot_df(const float4 &a, float sa, const float4 &b, float sb) {
    return df_add(df_add(df_prod(a.x * sa, b.x * sb), df_prod(a.y * sa, b.y * sb)), df_prod(a.z * sa, b.z * sb));
}

// a / b rounded to FP32 (a correction step on the FP32 quotient).
__device__ __forceinline__ float df_quotient(DFloat a, DFloat b) {
    const float q = __fdiv_rn(a.hi, b.hi);
    const float r = __fadd_rn(__fmaf_rn(-q, b.hi, a.hi), __fmaf_rn(-q, b.lo, a.lo));
    return isfinite(q) ? __fadd_rn(q, __fdiv_rn(r, b.hi)) : q;
}

// The power of two that brings a positive finite value to [1, 2) (1 for 0, or
// a non-finite one), within FP32's normal range.
__device__ __forceinline__ float unit_scale(float v) {
    if (!(v > 0.f) || !isfinite(v)) return 1.f;
    const int e = min(100, max(-100, ilogbf(v)));
    return __int_as_float((127 - e) << 23);
}

constexpr int kMaxWarps = 16;

struct Reduce {
    DFloat part[3][kMaxWarps], out[3];
};

// The sums (MAX: the maxima of .hi) of K values over every thread of every
// CTA, the same bits everywhere: a lane tree, the warps' totals in a lane tree,
// then the CTAs' words in a fixed order by one warp.  Every CTA writes its word
// to CG_COPIES places and reads one of them, so that no line is polled by all
// of them.  meanwhile(): work of every thread while the words travel.  Ends
// with a CTA barrier; false when a wait gave up.
template <int K, bool MAX, class F>
__device__ __forceinline__ bool all_reduce(DFloat (&v)[K], Reduce &sh, const CgArgs &a, unsigned tag, int &buf,
                                           bool ok, F meanwhile) {
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5, G = gridDim.x, c = blockIdx.x;
    float4 *words = a.red + (size_t)buf * 3 * CG_COPIES * G;
    buf ^= 1;
    auto join = [](DFloat x, DFloat y) { return MAX ? DFloat{fmaxf(x.hi, y.hi), 0.f} : df_add(x, y); };
    auto step = [&](DFloat x, int o) {
        return join(x, DFloat{__shfl_down_sync(full, x.hi, o), __shfl_down_sync(full, x.lo, o)});
    };
#pragma unroll
    for (int k = 0; k < K; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] = step(v[k], o);
        if (lane == 0) sh.part[k][w] = v[k];
    }
    __syncthreads();
    if (w == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            DFloat x = lane < W ? sh.part[k][lane] : DFloat{0.f, 0.f};
#pragma unroll
            for (int o = kMaxWarps / 2; o > 0; o >>= 1) x = step(x, o);
            x = DFloat{__shfl_sync(full, x.hi, 0), __shfl_sync(full, x.lo, 0)};
            const unsigned hi = __float_as_uint(x.hi), lo = __float_as_uint(x.lo);
            if (lane < CG_COPIES) st_word(words + ((size_t)k * CG_COPIES + lane) * G + c, hi, lo, hi ^ lo ^ tag, tag);
        }
        DFloat acc[K];
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] = DFloat{0.f, 0.f};
        const float4 *red = words + (size_t)(c % CG_COPIES) * G;
        constexpr int U = 5;  // 160 CTAs' words in flight at once
        for (int j0 = lane; j0 < G && ok; j0 += U * 32) {
            uint4 x[U][K];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int k = 0; k < K; ++k)
                    x[u][k] = j0 + 32 * u < G ? ld_word(red + (size_t)k * CG_COPIES * G + j0 + 32 * u)
                                              : make_uint4(0u, 0u, tag, tag);
            // (the check word ties the value to its tag: a sum that used a part
            // of the words only was compiled into narrower loads, and a maximum
            // paired a new tag with the last solve's value)
            auto whole = [&](const uint4 &v) { return v.w == tag && v.z == (v.x ^ v.y ^ tag); };
            Spin spin;
            for (;;) {
                bool ready = true;
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int k = 0; k < K; ++k) ready &= whole(x[u][k]);
                if (ready) break;
                if (spin.expired(a.err)) {
                    ok = false;
                    break;
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int k = 0; k < K; ++k)
                        if (!whole(x[u][k])) x[u][k] = ld_word(red + (size_t)k * CG_COPIES * G + j0 + 32 * u);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int k = 0; k < K; ++k)
                    acc[k] = join(acc[k], DFloat{__uint_as_float(x[u][k].x), __uint_as_float(x[u][k].y)});
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < K; ++k) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[k] = step(acc[k], o);
            if (lane == 0) sh.out[k] = acc[k];
        }
    }
    meanwhile();
    const bool all = !__syncthreads_or(!ok);
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = sh.out[k];
    return all;
}

// One CTA's view of its rows: vectors in shared memory where they fit, else in
// the workspace (generic pointers).
template <int NV, typename COL> struct Rows {
    float4 *P, *R, *Q, *X;  // direction (own rows, then the halo), residual, q (and z), solution
    const float *val;
    const COL *col;
    const int *node, *rlen, *soff;  // a row's padded node and length; a slice's first entry from the CTA's first
    const int *halo, *send;         // places of the halo's words; own rows that others read
    const float *dinv;              // NV values a row
    // (A v) of local row lr, v in P
    __device__ __forceinline__ float4 mul(int lr) const {
        const int s = lr >> 5, lane = lr & 31, n = rlen[lr];
        const size_t e0 = (size_t)soff[s];
        float sx = 0.f, sy = 0.f, sz = 0.f;
        const COL *cp = col + e0 * 32 + lane;
        const float *vp = val + e0 * (32 * NV) + lane;
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
            const float4 v = P[cp[32 * k]];
            if (NV == 1) {  // blocks a I3
                const float t = vp[32 * k];
                sx += t * v.x;
                sy += t * v.y;
                sz += t * v.z;
            } else {
                const float *t = vp + 32 * NV * k;
                sx += t[0] * v.x + t[32] * v.y + t[64] * v.z;
                sy += t[96] * v.x + t[128] * v.y + t[160] * v.z;
                sz += t[192] * v.x + t[224] * v.y + t[256] * v.z;
            }
        }
        return f4(sx, sy, sz);
    }
};

template <int NV, typename COL, int PER_SM>
__global__ void __launch_bounds__(512, PER_SM) k_cg_solve(CgPlanView pl, CgArgs a) {
    extern __shared__ float4 smem4[];
    __shared__ Reduce sh;
    char *sm = reinterpret_cast<char *>(smem4);
    const int c = blockIdx.x, tid = threadIdx.x, T = blockDim.x;
    const int s0 = pl.cta_slice[c], ns = pl.cta_slice[c + 1] - s0, nr = pl.cta_rows[c];
    const int h0 = pl.cta_halo[c], nh = pl.cta_halo[c + 1] - h0;
    const int d0 = pl.cta_send[c], nd = pl.cta_send[c + 1] - d0;
    float4 *words = a.xp + 32 * (size_t)s0;  // this CTA's own
    Rows<NV, COL> L;
    {
        const size_t rb = 32 * (size_t)s0;
        const size_t e0 = (size_t)pl.soff[s0], ne = (size_t)pl.soff[s0 + ns] - e0;
        // a constant array: copied to shared memory where it has a place there
        auto keep = [&](int off, const void *src, size_t bytes) -> const void * {
            if (off < 0) return src;
            float4 *d = reinterpret_cast<float4 *>(sm + off);
            const float4 *q = reinterpret_cast<const float4 *>(src);
            for (size_t j = tid; j < bytes / 16; j += T) cp_async16(d + j, q + j);
            return d;
        };
        auto place = [&](int off, float4 *global) { return off >= 0 ? reinterpret_cast<float4 *>(sm + off) : global; };
        L.node = (const int *)keep(pl.off_node, pl.srow + rb, 128 * (size_t)ns);
        L.rlen = (const int *)keep(pl.off_rlen, pl.rlen + rb, 128 * (size_t)ns);
        L.val = (const float *)keep(pl.off_val, a.val + e0 * (32 * NV), ne * (128 * NV));
        L.col = (const COL *)keep(pl.off_col, reinterpret_cast<const COL *>(pl.scol) + e0 * 32, ne * (32 * sizeof(COL)));
        L.soff = pl.soff_local + s0;
        L.halo = pl.halo + h0;
        L.send = pl.send + d0;
        L.dinv = a.dinv + rb * NV;
        if (pl.off_small >= 0) {  // the unaligned ones
            int *d = reinterpret_cast<int *>(sm + pl.off_small);
            for (int j = tid; j < ns; j += T) d[j] = L.soff[j];
            for (int j = tid; j < nh; j += T) d[ns + j] = L.halo[j];
            for (int j = tid; j < nd; j += T) d[ns + nh + j] = L.send[j];
            L.soff = d;
            L.halo = d + ns;
            L.send = d + ns + nh;
        }
        L.dinv = (const float *)keep(pl.off_dinv, a.dinv + rb * NV, 128 * (size_t)ns * NV);
        L.P = place(pl.off_p, a.ws_p + rb + h0);
        L.R = place(pl.off_r, a.ws_r + rb);
        L.Q = place(pl.off_q, a.ws_q + rb);
        L.X = place(pl.off_x, a.ws_x + rb);
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
    }
    unsigned tag = *a.tag;  // (this launch's own tags follow; CTA 0 writes the last back at the end)
    int buf = 0;
    bool ok = true;
    // the words of the own rows that others read out, the halo's in
    auto exchange = [&]() {
        ++tag;
        __syncthreads();  // P is written by its rows' threads
        for (int j = tid; j < nd; j += T) {
            const int lr = L.send[j];
            const float4 v = L.P[lr];
            st_word(words + lr, make_float3(v.x, v.y, v.z), tag);
        }
        constexpr int U = 4;  // words in flight a thread
        for (int j0 = tid; j0 < nh; j0 += U * T) {
            const float4 *p[U];
            uint4 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                p[u] = j0 + u * T < nh ? a.xp + L.halo[j0 + u * T] : nullptr;
                v[u] = make_uint4(0u, 0u, 0u, tag);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (p[u]) v[u] = ld_word(p[u]);
            Spin spin;
            for (;;) {
                bool ready = true;
#pragma unroll
                for (int u = 0; u < U; ++u) ready &= v[u].w == tag;
                if (ready) break;
                if (spin.expired(a.err)) {
                    ok = false;
                    break;
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (v[u].w != tag) v[u] = ld_word(p[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (p[u]) L.P[nr + j0 + u * T] = word_f4(v[u]);
        }
        ok = !__syncthreads_or(!ok);
    };
    auto dinv = [&](int lr, const float4 &r) {
        const float *D = L.dinv + (lr >> 5) * (32 * NV) + (lr & 31);
        if (NV == 1) return f4(D[0] * r.x, D[0] * r.y, D[0] * r.z);
        return f4(D[0] * r.x + D[32] * r.y + D[64] * r.z, D[96] * r.x + D[128] * r.y + D[160] * r.z,
                  D[192] * r.x + D[224] * r.y + D[256] * r.z);
    };

    // r = b - A x, z = D^-1 r, p = z
    for (int lr = tid; lr < nr; lr += T) L.P[lr] = L.X[lr] = a.x[L.node[lr]];
    exchange();
    float mr = 0.f, mz = 0.f;
    for (int lr = tid; lr < nr && ok; lr += T) {
        const float4 ax = L.mul(lr), b = a.b[L.node[lr]];
        const float4 r = f4(b.x - ax.x, b.y - ax.y, b.z - ax.z);
        const float4 z = dinv(lr, r), db = dinv(lr, b);
        L.R[lr] = r;
        L.Q[lr] = z;
        auto top = [](float m, const float4 &v) {
            return fmaxf(m, fmaxf(fabsf(v.x), fmaxf(fabsf(v.y), fabsf(v.z))));
        };
        mr = top(top(mr, r), b);
        mz = top(top(mz, z), db);
    }
    DFloat mx[2] = {DFloat{mr, 0.f}, DFloat{mz, 0.f}};
    ok = ok && all_reduce<2, true>(mx, sh, a, ++tag, buf, ok, [] {});
    const float sr = unit_scale(mx[0].hi), sz = unit_scale(mx[1].hi);
    DFloat in[3] = {DFloat{0.f, 0.f}, DFloat{0.f, 0.f}, DFloat{0.f, 0.f}};  // r.z, r.r, b.b or b.D^-1 b
    for (int lr = tid; lr < nr && ok; lr += T) {
        const float4 r = L.R[lr], z = L.Q[lr], b = a.b[L.node[lr]];
        in[0] = df_add(in[0], dot_df(r, sr, z, sz));
        in[1] = df_add(in[1], dot_df(r, sr, r, sr));
        in[2] = df_add(in[2], a.pnorm ? dot_df(b, sr, dinv(lr, b), sz) : dot_df(b, sr, b, sr));
        L.P[lr] = z;
    }
    ok = ok && all_reduce<3, false>(in, sh, a, ++tag, buf, ok, [] {});
    DFloat rz = in[0], rr = in[1];
    const double lim = a.tol2 * df_double(in[2]);
    const float lim_hi = (float)lim, lim_lo = (float)(lim - (double)lim_hi);
    auto below = [&](DFloat v) { return v.hi < lim_hi || (v.hi == lim_hi && v.lo <= lim_lo); };
    int iters = 0, status = PBS_OK;
    bool done = below(a.pnorm ? rz : rr);  // the initial guess already solves it
    if (!done && !isfinite(rr.hi + rr.lo)) {
        status = PBS_E_NONFINITE;
        done = true;
    }
    while (ok && !done) {
        exchange();
        if (!ok) break;
        // q = A p, alpha = r.z / p.q
        DFloat pq[1] = {DFloat{0.f, 0.f}};
        for (int lr = tid; lr < nr; lr += T) {
            const float4 q = L.mul(lr);
            L.Q[lr] = q;
            pq[0] = df_add(pq[0], dot_df(L.P[lr], sz, q, sr));
        }
        ok = all_reduce<1, false>(pq, sh, a, ++tag, buf, ok, [] {});
        if (!ok) break;
        const float alpha = pq[0].hi != 0.f ? df_quotient(rz, pq[0]) : 0.f;
        if (!isfinite(alpha) || !(pq[0].hi > 0.f)) {
            status = PBS_E_NONFINITE;
            break;
        }
        // r -= alpha q, z = D^-1 r; x += alpha p while the sums travel
        auto add_x = [&] {
            for (int lr = tid; lr < nr; lr += T) {
                const float4 p = L.P[lr], x = L.X[lr];
                L.X[lr] = f4(x.x + alpha * p.x, x.y + alpha * p.y, x.z + alpha * p.z);
            }
        };
        DFloat d[2] = {DFloat{0.f, 0.f}, DFloat{0.f, 0.f}};
        for (int lr = tid; lr < nr; lr += T) {
            const float4 q = L.Q[lr], r0 = L.R[lr];
            const float4 r = f4(r0.x - alpha * q.x, r0.y - alpha * q.y, r0.z - alpha * q.z);
            const float4 z = dinv(lr, r);
            L.R[lr] = r;
            L.Q[lr] = z;
            d[0] = df_add(d[0], dot_df(r, sr, z, sz));
            if (!a.pnorm) d[1] = df_add(d[1], dot_df(r, sr, r, sr));
        }
        ++iters;
        if (a.pnorm) {  // (one sum: a non-finite r shows in r.z)
            DFloat e[1] = {d[0]};
            ok = all_reduce<1, false>(e, sh, a, ++tag, buf, ok, add_x);
            d[0] = d[1] = e[0];
        } else {
            ok = all_reduce<2, false>(d, sh, a, ++tag, buf, ok, add_x);
        }
        if (!ok) break;
        const float beta = rz.hi != 0.f ? df_quotient(d[0], rz) : 0.f;
        rz = d[0];
        rr = d[1];
        if (!isfinite(rr.hi + rr.lo)) {
            status = PBS_E_NONFINITE;
            break;
        }
        if (below(rr)) break;
        if (iters >= a.max_iters) {
            status = PBS_E_ITER_CAP;
            break;
        }
        // p = z + beta p
        for (int lr = tid; lr < nr; lr += T) {
            const float4 z = L.Q[lr], p = L.P[lr];
            L.P[lr] = f4(z.x + beta * p.x, z.y + beta * p.y, z.z + beta * p.z);
        }
    }
    for (int lr = tid; lr < nr && ok; lr += T) a.x[L.node[lr]] = L.X[lr];
    if (c == 0 && tid == 0) {
        CgState s;
        const double ir = 1.0 / (double)sr, iz = 1.0 / (double)sz;
        s.rz = df_double(rz) * ir * iz;
        s.rr = df_double(rr) * ir * ir;
        s.bb = df_double(in[2]) * ir * (a.pnorm ? iz : ir);
        s.iters = iters;
        s.status = ok ? status : PBS_E_DEVICE_TIMEOUT;
        *a.cs = s;
        *a.tag = tag;  // every CTA has read it: each gave a word to the first sum
    }
}

// CTAs a SM of the solve beside others (CgPlanView::light).  Eight threads, one
// handle each, us a step of all, in turn / two a SM with 110 KB / three with 73:
// projective dynamics of 100,000 tets 2250 / 2143 / 1842, 200,000 5800 / 4383 /
// 3960, 500,000 (10,430) / 8245 / 7629; backward Euler, two a SM with 110 KB /
// with 55 (the matrix from L2) / three with 73: 100,000 3054 / 2373 / 2612,
// 200,000 5342 / 5256 / 5993.
template <int NV> constexpr int LIGHT_PER_SM = NV == 1 ? 3 : 2;

template <int NV, typename COL, int PER_SM>
cudaError_t launch_solve_t(cudaStream_t s, const CgPlanView &pl, const CgArgs &a) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.grid);
    cfg.blockDim = dim3(pl.threads);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_cg_solve<NV, COL, PER_SM>, pl, a);
}

template <int NV, typename COL> cudaError_t launch_solve_p(cudaStream_t s, const CgPlanView &pl, const CgArgs &a) {
    return pl.light ? launch_solve_t<NV, COL, LIGHT_PER_SM<NV>>(s, pl, a) : launch_solve_t<NV, COL, 1>(s, pl, a);
}

}  // namespace

cudaError_t launch_bsr_count(cudaStream_t s, const DevMesh &m, int *cnt) {
    k_bsr_count<<<(m.Np + 127) / 128, 128, 0, s>>>(m, cnt);
    return cudaGetLastError();
}
cudaError_t launch_bsr_fill(cudaStream_t s, const DevMesh &m, const int *ptr, int *col) {
    k_bsr_fill<<<(m.Np + 127) / 128, 128, 0, s>>>(m, ptr, col);
    return cudaGetLastError();
}
cudaError_t launch_cg_pack(cudaStream_t s, const CgPlanView &pl, const BsrView &A, const float *dinv9, float *out,
                           float *dinv) {
    const int g = (pl.n_slices + 7) / 8;
    if (A.scalar) k_cg_pack<1><<<g, 256, 0, s>>>(pl, A, dinv9, out, dinv);
    else k_cg_pack<9><<<g, 256, 0, s>>>(pl, A, dinv9, out, dinv);
    return cudaGetLastError();
}
template <int NV, typename COL> static cudaError_t allow_cg() {
    const cudaError_t e = allow_all_smem(k_cg_solve<NV, COL, 1>);
    return e != cudaSuccess ? e : allow_all_smem(k_cg_solve<NV, COL, LIGHT_PER_SM<NV>>);
}
cudaError_t prepare_cg_kernels() {
    const cudaError_t e[] = {allow_cg<1, int>(), allow_cg<9, int>(), allow_cg<1, unsigned short>(),
                             allow_cg<9, unsigned short>()};
    for (cudaError_t x : e)
        if (x != cudaSuccess) return x;
    return cudaSuccess;
}
cudaError_t launch_cg_solve(cudaStream_t s, const CgPlanView &pl, const CgArgs &a, bool scalar) {
    if (pl.col32) return scalar ? launch_solve_p<1, int>(s, pl, a) : launch_solve_p<9, int>(s, pl, a);
    return scalar ? launch_solve_p<1, unsigned short>(s, pl, a) : launch_solve_p<9, unsigned short>(s, pl, a);
}

}  // namespace pbs

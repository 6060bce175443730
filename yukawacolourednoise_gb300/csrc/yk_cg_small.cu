// yk_cg_small.cu -- the CG on D^dag D (or D D^dag) of code/src/CGsolver.cu:72-170
// inside one thread-block cluster per system, for lattices whose vectors fit the
// shared memory of at most 16 SMs: every FP64 solve and every complex solve
// (caller-given sources, pions) of a small lattice.  The iteration, its stopping
// rule and the mixed solver's reliable updates are those of cg_kernel (yk_cg.cu).
//
// What bounds a small solve is latency: cg_kernel spends a neighbour sync, a grid
// barrier and two round trips through L2 per iteration, and at FP64 (1/64 of the
// FP32 rate on GB300) it forms r and p at five sites per site.  Microseconds an
// iteration, cg_kernel and here: FP64 real 23.1 and 3.9 at 32 x 32, 23.3 and 8.1 at
// 64 x 64, 23.5 and 19.5 at 128 x 96.  (With remote stores and two cluster barriers an
// iteration: 4.4, 8.5 and 19.9; FP64 complex, 32 x 32: 36.9 and 5.9; mixed complex: 12.4
// and 3.7 at 64 x 64, 12.4 and 7.2 at 128 x 128.)  Here a CTA owns a contiguous range of sites and keeps
//   p, r, t = D_first p   in shared memory, on its sites and the Nx before and after,
//   x (or the FP32 increment) and A p   of its own sites in registers,
// and an iteration exchanges twice, by asynchronous stores counted on mbarriers:
//   T: t = D_first p on the own sites; the edge sites' t is also stored into the
//      neighbours' shared memory                          -> neighbours
//   B: A p = D_second t, its edges stored into the neighbours, the four sums'
//      partials into every CTA of the cluster             -> every CTA
//   U: every CTA sums the partials in the same order and runs the same scalar
//      step, then updates r and p on its own sites and, with the neighbours' A p,
//      on the sites around them (redundantly: no third exchange).
// All exchange is by remote stores, all loads are local.
//
// A thread works on one flavour of a site (both spin entries, K planes): the
// operator does not mix flavours (the pions' term reads the other one's entries).
// At r = 1 the time hops keep one spin entry each and the space hops share their
// sums: 8 operations per spin pair against 14 in the general form, and half the
// time neighbours' loads.  Four sums cost 6 additions per warp and lane (each
// halving of the warp also halves the values a lane carries) against 20.
#include <cfloat>
#include <type_traits>

#include "yk_cluster.cuh"
#include "yk_kernels.h"

namespace yk {

namespace {

constexpr int kSmMaxC = 16;
constexpr int kSmThreads = 512;
constexpr size_t kSmMaxSmem = 220 * 1024;
constexpr int kSmMaxReal = 12288;   // sites of a real FP64 solve (small_form)

// FP64 data of global memory that another CTA of the cluster wrote before the
// last barrier: served by L2.
template <int K>
__device__ __forceinline__ Unit<double, K> ld_unit64(const double* base, int i)
{
    Unit<double, K> s;
#pragma unroll
    for (int q = 0; q < K; ++q)
        asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];"
                     : "=d"(s.v[2 * q]), "=d"(s.v[2 * q + 1])
                     : "l"(base + (size_t)i * 2 * K + 2 * q)
                     : "memory");
    return s;
}

// Offsets (in units) of a unit's neighbours and the signs of its time hops.
struct Hop {
    int tu, td, xu, xd;
    bool np, nm;   // the hop to t + 1 (t - 1) changes sign
};

// D (s = 1) or D^dag (s = -1) at unit i of `at` (dirac_combine, yk_common.cuh):
// r = 1 keeps the time hops -D: d of t + 1, u of t - 1; D^dag the others.
template <typename W, int K, typename At>
__device__ __forceinline__ Unit<W, K> unit_dirac(const At& at, int i, const Hop& h, W diag, W r, W s)
{
    const Unit<W, K> c = at(i), xu = at(i + h.xu), xd = at(i + h.xd);
    const W half = W(0.5);
    const W sp = h.np ? W(-1) : W(1), sm = h.nm ? W(-1) : W(1);
    Unit<W, K> o;
    if (r == W(1)) {
        const bool dag = s < W(0);
        const Unit<W, K> tu = at(i + (dag ? h.tu : h.td)), td = at(i + (dag ? h.td : h.tu));
        const W su = dag ? sp : sm, sd = dag ? sm : sp;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const W a = fma(-s, xu.v[K + k], xu.v[k]), b = fma(s, xd.v[K + k], xd.v[k]);
            o.v[k] = fma(-half, a + b, fma(diag, c.v[k], -su * tu.v[k]));
            o.v[K + k] = fma(half * s, a - b, fma(diag, c.v[K + k], -sd * td.v[K + k]));
        }
    } else {
        const Unit<W, K> tu = at(i + h.tu), td = at(i + h.td);
        const W uu = -sp * half * (r - s), ud = -sp * half * (r + s), du = -sm * half * (r + s),
                dd = -sm * half * (r - s), ax = -half * r, bx = half * s;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            W ou = diag * c.v[k], od = diag * c.v[K + k];
            ou = fma(uu, tu.v[k], fma(du, td.v[k], ou));
            od = fma(ud, tu.v[K + k], fma(dd, td.v[K + k], od));
            ou = fma(bx, xu.v[K + k] - xd.v[K + k], fma(ax, xu.v[k] + xd.v[k], ou));
            od = fma(bx, xu.v[k] - xd.v[k], fma(ax, xu.v[K + k] + xd.v[K + k], od));
            o.v[k] = ou;
            o.v[K + k] = od;
        }
    }
    return o;
}

enum SmMode { kSmStep = 1, kSmRu = 2, kSmRedo = 3, kSmDone = 4 };

// The solve's scalar state, the same bits in every CTA (warp 0 computes it).
struct SmState {
    double rr, rr0, rr_prev, stop2, rmax2;
    double alpha, beta, c_re, c_im;
    int mode, iters, n_ru, status, converged, ru;
};

}  // namespace

// W: the iteration's arithmetic (double: FP64 CG; float: mixed), U: units a
// thread owns at most.
template <typename W, int K, int U>
__global__ void __launch_bounds__(kSmThreads, 1) cg_small_kernel(CGArgs a, int pions)
{
    constexpr bool MIXED = sizeof(W) == 4;
    using T = typename std::conditional<MIXED, FF, double>::type;
    using Un = Unit<W, K>;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    __shared__ T wred[kSmThreads / 32][4];
    __shared__ __align__(8) T cpart[2][kSmMaxC][4];   // by the iteration's parity
    __shared__ __align__(8) uint64_t mb[4];           // arrivals: t and A p around, cpart[0], cpart[1]
    __shared__ int s_dead, s_left;                    // a wait gave up; CTAs that then came to the end
    __shared__ SmState st;
    unsigned rank, nc;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(nc));
    const int tid = threadIdx.x, TB = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = TB >> 5;
    const int sys = a.sys_first + (int)(blockIdx.x / nc);
    const SysDev& S = a.sys[sys];
    const int Nt = S.Nt, Nx = S.Nx, V = S.V;
    const int n0 = (int)((int64_t)V * rank / nc), n1 = (int)((int64_t)V * (rank + 1) / nc), own = n1 - n0;
    const unsigned next = rank + 1 == nc ? 0 : rank + 1, prev = rank == 0 ? nc - 1 : rank - 1;
    const int prev_own = (int)((int64_t)V * (prev + 1) / nc) - (int)((int64_t)V * prev / nc);
    const int omax = (V + (int)nc - 1) / (int)nc, span = 2 * (omax + 2 * Nx);   // units of a buffer
    Un* const sp = reinterpret_cast<Un*>(sm_raw);
    Un* const sr = sp + span;
    Un* const stt = sr + span;
    Un* const sa = stt + span;                       // A p on the sites around: before, after
    W* const sdiag = reinterpret_cast<W*>(sa + 4 * Nx);
    W* const spi = sdiag + omax;                     // g pi_a, when the chain carries pions
    const unsigned t_next = cta_addr(stt, next), t_prev = cta_addr(stt + 2 * (Nx + prev_own), prev);
    const unsigned a_next = cta_addr(sa, next), a_prev = cta_addr(sa + 2 * Nx, prev);
    const unsigned mb0 = (unsigned)__cvta_generic_to_shared(mb), mb_next = cta_addr(mb, next), mb_prev = cta_addr(mb, prev);
    const bool first_dag = (a.mtype == YK_NORMAL);   // Normal: A = D D^dag, apply D^dag first
    const W s1st = first_dag ? W(-1) : W(1);
    const W r = (W)S.r;
    const int units = 2 * own;

    // ---------------- round 0: x = 0, r = p = b on the own sites and around them
    for (int i = tid; i < 2 * (own + 2 * Nx); i += TB) {
        const int l = (i >> 1) - Nx, f = i & 1;
        int n = n0 + l;
        n = n < 0 ? n + V : (n >= V ? n - V : n);
        Unit<double, K> b;
        if (S.gen_eta) {
            const Site<double, K> e = eta_of_step<K>(S, n, a.eta_kind);
#pragma unroll
            for (int q = 0; q < 2 * K; ++q) b.v[q] = f ? e.v[2 * K + q] : e.v[q];
        } else {
            b = reinterpret_cast<const Unit<double, K>*>(S.b)[2 * (size_t)n + f];
        }
        Un w;
#pragma unroll
        for (int q = 0; q < 2 * K; ++q) w.v[q] = (W)b.v[q];
        sp[i] = w;
        sr[i] = w;
        if (l >= 0 && l < own) {
            if (S.gen_eta) reinterpret_cast<Unit<double, K>*>(S.b)[2 * (size_t)n + f] = b;
            if constexpr (MIXED) {
                Unit<double, K> z;
#pragma unroll
                for (int q = 0; q < 2 * K; ++q) z.v[q] = 0.0;
                reinterpret_cast<Unit<double, K>*>(S.x)[2 * (size_t)n + f] = z;
            }
            if (f == 0) {
                sdiag[l] = (W)(2.0 * S.r + S.m0 + S.g * S.sigma[n]);
                if (K == 2 && pions)
#pragma unroll
                    for (int q = 0; q < 3; ++q) spi[q * omax + l] = (W)(S.g * S.pi[(size_t)q * V + n]);
            }
        }
    }
    Un x[U], ap[U];
    unsigned edge = 0;   // four flags per unit: x wraps upwards, downwards; t + 1, t - 1 change sign
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int i = tid + u * TB;
#pragma unroll
        for (int q = 0; q < 2 * K; ++q) x[u].v[q] = ap[u].v[q] = W(0);
        if (i < units) {
            const int n = n0 + (i >> 1), t = n / Nx, xx = n - t * Nx;
            edge |= (unsigned)((xx + 1 == Nx ? 1 : 0) | (xx == 0 ? 2 : 0) | (t + 1 == Nt ? 4 : 0) | (t == 0 ? 8 : 0))
                    << (4 * u);
        }
    }
    auto hop = [&](int u) {
        const unsigned e = edge >> (4 * u);
        Hop h;
        h.tu = 2 * Nx;
        h.td = -2 * Nx;
        h.xu = (e & 1) ? 2 - 2 * Nx : 2;
        h.xd = (e & 2) ? 2 * Nx - 2 : -2;
        h.np = e & 4;
        h.nm = e & 8;
        return h;
    };
    // D_first or D_second of a shared-memory vector at the thread's unit u
    auto apply = [&](const Un* buf, int u, W s) {
        const int i = tid + u * TB, l = i >> 1, f = i & 1, j = i + 2 * Nx;
        Un o = unit_dirac<W, K>([&](int q) { return buf[q]; }, j, hop(u), sdiag[l], r, s);
        if constexpr (K == 2)
            if (pions) unit_pions<W>(o, buf[j], buf[j ^ 1], f, s * spi[l], s * spi[omax + l], s * spi[2 * omax + l]);
        return o;
    };
    // many units a thread: their loads do not all go ahead of the first one's
    // arithmetic (that spilled)
    auto unit_end = [] {
        if constexpr (U >= 4) asm volatile("" ::: "memory");
    };
    // the four sums of the CTA's values into every CTA's cpart
    auto partials = [&](const auto& v, int b, bool async) {
        const auto c = warp_sum4(v);
        if ((lane & 7) == 0) wred[warp][lane >> 3] = s_of(c, T{});
        __syncthreads();
        if (warp == 0) {
            const int v4 = lane >> 3, w0 = lane & 7;
            T t = w0 < nw ? wred[w0][v4] : s_zero(T{});
            if (w0 + 8 < nw) t = s_add(t, wred[w0 + 8][v4]);
            t = s_add(t, s_shfl(t, 4));
            t = s_add(t, s_shfl(t, 2));
            t = s_add(t, s_shfl(t, 1));
            for (unsigned c2 = w0; c2 < nc; c2 += 8)
                if (async)
                    st_async(cta_addr(&cpart[b][rank][v4], c2), t, cta_addr(mb + 2 + b, c2));
                else
                    *in_cta(&cpart[b][rank][v4], c2) = t;
        }
    };
    // the cluster's sums, in every lane of warp 0
    auto totals = [&](double (&s)[4], int b) {
        const int v4 = lane >> 3, w0 = lane & 7;
        T t = w0 < (int)nc ? cpart[b][w0][v4] : s_zero(T{});
        if (w0 + 8 < (int)nc) t = s_add(t, cpart[b][w0 + 8][v4]);
        t = s_add(t, s_shfl(t, 4));
        t = s_add(t, s_shfl(t, 2));
        t = s_add(t, s_shfl(t, 1));
        const double d = s_val(t);
#pragma unroll
        for (int q = 0; q < 4; ++q) s[q] = __shfl_sync(0xffffffffu, d, 8 * q);
    };
    if (tid == 0) {
        st.rr = st.rr0 = st.rr_prev = st.stop2 = st.rmax2 = st.alpha = st.beta = st.c_im = 0.0;
        st.c_re = 1.0;
        st.mode = kSmStep;
        st.iters = st.n_ru = st.status = st.converged = st.ru = 0;
        if (blockIdx.x == 0) *a.err = 0;   // (the solve's one launch: another CTA's wait gives up 2 s later)
        s_dead = s_left = 0;
        for (int q = 0; q < 4; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb0 + 8u * q) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster_barrier();   // every CTA of the cluster has started: its shared memory can be written

    // (How far apart CTAs can be: one sends the t of iteration k + 1 with every CTA's
    // sums of iteration k, each sent after that CTA's last use of t_k, and A p of k + 1
    // with the neighbours' t of k + 1, sent after they used A p of k; the sums
    // alternate between two places.)
    for (int k = 0;; ++k) {
        const int par = k & 1;
        if (tid == 0) {
            mb_expect(mb0, 4u * (unsigned)Nx * (unsigned)sizeof(Un));
            mb_expect(mb0 + 8, 4u * (unsigned)Nx * (unsigned)sizeof(Un));
            mb_expect(mb0 + 16 + 8 * par, 32u * nc);
        }
        // ---------------- T
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = tid + u * TB;
            if (i < units) {
                const Un t = apply(sp, u, s1st);
                stt[i + 2 * Nx] = t;
                if (i < 2 * Nx) st_async16(t_prev + (unsigned)(i * sizeof(Un)), t, mb_prev);
                if (i >= units - 2 * Nx) st_async16(t_next + (unsigned)((i - (units - 2 * Nx)) * sizeof(Un)), t, mb_next);
            }
            unit_end();
        }
        __syncthreads();
        mb_wait(mb0, par, &s_dead);
        // ---------------- B
        W v[4] = {W(0), W(0), W(0), W(0)};
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = tid + u * TB;
            if (i < units) {
                ap[u] = apply(stt, u, -s1st);
                if (i < 2 * Nx) st_async16(a_prev + (unsigned)(i * sizeof(Un)), ap[u], mb_prev + 8);
                if (i >= units - 2 * Nx) st_async16(a_next + (unsigned)((i - (units - 2 * Nx)) * sizeof(Un)), ap[u], mb_next + 8);
                const Un rv = sr[i + 2 * Nx], pv = sp[i + 2 * Nx];
#pragma unroll
                for (int q = 0; q < 2 * K; ++q) {
                    v[0] = fma(rv.v[q], rv.v[q], v[0]);
                    v[1] = fma(ap[u].v[q], ap[u].v[q], v[1]);
                    v[2] = fma(pv.v[q], ap[u].v[q], v[2]);
                    v[3] = fma(rv.v[q], ap[u].v[q], v[3]);
                }
            }
            unit_end();
        }
        partials(v, par, true);
        // ---------------- the scalar step (scalar_step, yk_cg.cu; A is Hermitian, so
        // <p, A p> and alpha are real)
        if (warp == 0) {
            mb_wait(mb0 + 16 + 8 * par, (k >> 1) & 1, &s_dead);
            double s[4];
            totals(s, par);
            const double rr = s[0];
            SmState q = st;
            q.rr = rr;
            q.iters = k;
            q.ru = 0;
            if (k == 0) {
                q.stop2 = (a.tol_mode == YK_TOL_ABS) ? a.tol * a.tol : a.tol * a.tol * rr;
                q.rmax2 = q.rr0 = rr;
            }
            double alpha, inv_rr = 0.0;
            if constexpr (MIXED) {
                alpha = (double)(1.f / ((float)s[2] * (1.f / (float)rr)));
            } else {
                // both divisions at once, in different lanes
                const double d = (lane & 1 ? 1.0 : rr) / (lane & 1 ? rr : s[2]);
                alpha = __shfl_sync(0xffffffffu, d, 0);
                inv_rr = __shfl_sync(0xffffffffu, d, 1);
            }
            q.mode = kSmDone;
            if (*(volatile int*)&s_dead) {
                q.status = YK_ETIMEOUT;
                if (lane == 0) *a.err = YK_ETIMEOUT;
            } else if (!isfinite(rr)) {
                q.status = YK_ENAN;
            } else if ((!MIXED || k == 0) && !(rr > q.stop2)) {
                q.converged = 1;
            } else if (k >= a.max_iter) {
                q.status = YK_ENOCONV;
            } else if (!isfinite(alpha)) {
                q.status = YK_ENAN;
            } else {
                // |r - alpha A p|^2
                double est = fma(-alpha, fma(-alpha, s[1], 2.0 * s[3]), rr);
                if (!(est > 0.0)) est = 0.0;
                q.rr_prev = rr;
                q.alpha = alpha;
                q.mode = kSmStep;
                if constexpr (MIXED) {
                    q.beta = (double)((float)est / (float)rr);
                    q.rmax2 = fmax(q.rmax2, rr);
                    const bool cand = !(rr > q.stop2) || !(est > q.stop2);
                    const bool drop = est < a.reliable_delta * a.reliable_delta * q.rmax2;
                    const bool due = a.reliable_every > 0 && (k + 1) % a.reliable_every == 0;
                    if (cand || drop || due || k + 1 >= a.max_iter) q.mode = kSmRu;
                } else {
                    q.beta = est * inv_rr;
                }
            }
            __syncwarp();
            if (lane == 0) st = q;
        }
        __syncthreads();
        mb_wait(mb0 + 8, par, &s_dead);   // also at the end: nothing may come in after it
        if (st.mode == kSmDone) break;
        const W alpha = (W)st.alpha;
        W beta = (W)st.beta, cre = W(1), cim = W(0);
        if constexpr (MIXED) {
            if (st.mode == kSmRu) {
                // ---------------- reliable update of x_{k+1}, in FP64 through global memory:
                // x += increment + alpha p, t64 = D_first x, r = b - D_second t64
                const double al = st.alpha;
                const double s1 = first_dag ? -1.0 : 1.0;
                double* const gx = S.x;
                double* const gt = S.t64;
                auto ghop = [&](int u) {
                    const unsigned e = edge >> (4 * u);
                    Hop h = hop(u);
                    if (e & 4) h.tu = -2 * Nx * (Nt - 1);
                    if (e & 8) h.td = 2 * Nx * (Nt - 1);
                    return h;
                };
                auto gapply = [&](const double* buf, int u, double s) {
                    const int i = tid + u * TB, n = n0 + (i >> 1), f = i & 1, j = 2 * n + f;
                    const double diag = 2.0 * S.r + S.m0 + S.g * S.sigma[n];
                    Unit<double, K> o = unit_dirac<double, K>([&](int q) { return ld_unit64<K>(buf, q); }, j, ghop(u),
                                                              diag, S.r, s);
                    if constexpr (K == 2)
                        if (pions) {
                            const double g = s * S.g;
                            unit_pions<double>(o, ld_unit64<K>(buf, j), ld_unit64<K>(buf, j ^ 1), f, g * S.pi[n],
                                               g * S.pi[(size_t)V + n], g * S.pi[2 * (size_t)V + n]);
                        }
                    return o;
                };
#pragma unroll 1
                for (int u = 0; u < U; ++u) {
                    const int i = tid + u * TB;
                    if (i < units) {
                        Unit<double, K>* g = reinterpret_cast<Unit<double, K>*>(gx) + 2 * (size_t)n0 + i;
                        Unit<double, K> xv = *g;
                        const Un p = sp[i + 2 * Nx];
                        Un inc;
#pragma unroll
                        for (int w = 0; w < U; ++w)
                            if (w == u) {
                                inc = x[w];
#pragma unroll
                                for (int q = 0; q < 2 * K; ++q) x[w].v[q] = W(0);
                            }
#pragma unroll
                        for (int q = 0; q < 2 * K; ++q)
                            xv.v[q] = fma(al, (double)p.v[q], xv.v[q] + (double)inc.v[q]);
                        *g = xv;
                    }
                }
                cluster_barrier();
#pragma unroll 1
                for (int u = 0; u < U; ++u) {
                    const int i = tid + u * TB;
                    if (i < units) reinterpret_cast<Unit<double, K>*>(gt)[2 * (size_t)n0 + i] = gapply(gx, u, s1);
                }
                cluster_barrier();
                double w4[4] = {0.0, 0.0, 0.0, 0.0};
                Un* const r_next = in_cta(sr, next);
                Un* const r_prev = in_cta(sr, prev) + 2 * (Nx + prev_own);
#pragma unroll 1
                for (int u = 0; u < U; ++u) {
                    const int i = tid + u * TB;
                    if (i < units) {
                        const Unit<double, K> ax = gapply(gt, u, -s1);
                        const Unit<double, K> b = reinterpret_cast<const Unit<double, K>*>(S.b)[2 * (size_t)n0 + i];
                        const Un p = sp[i + 2 * Nx];
                        Un rw;
                        double e[2 * K];
#pragma unroll
                        for (int q = 0; q < 2 * K; ++q) {
                            e[q] = b.v[q] - ax.v[q];
                            rw.v[q] = (W)e[q];
                            w4[0] = fma(e[q], e[q], w4[0]);
                            w4[2] = fma(e[q], (double)p.v[q], w4[2]);
                        }
                        if constexpr (K == 2)
#pragma unroll
                            for (int q = 0; q < 4; q += 2)
                                w4[3] += e[q] * (double)p.v[q + 1] - e[q + 1] * (double)p.v[q];
                        sr[i + 2 * Nx] = rw;
                        if (i < 2 * Nx) r_prev[i] = rw;
                        if (i >= units - 2 * Nx) r_next[i - (units - 2 * Nx)] = rw;
                    }
                }
                T f4[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) f4[q] = s_of(w4[q], T{});
                partials(f4, par, false);
                cluster_barrier();
                if (warp == 0) {
                    double s[4];
                    totals(s, par);
                    SmState q = st;
                    const double rr = s[0];
                    q.rr = rr;
                    q.iters = k + 1;
                    q.n_ru += 1;
                    q.ru = 1;
                    q.mode = kSmDone;
                    if (!isfinite(rr)) {
                        q.status = YK_ENAN;
                    } else if (!(rr > q.stop2)) {
                        q.converged = 1;
                    } else if (k + 1 >= a.max_iter) {
                        q.status = YK_ENOCONV;
                    } else {
                        // p = r + beta (p - gamma r), gamma = <r, p> / |r|^2; the
                        // divisions in FP32 where its range allows (scalar_step)
                        const float rf = (float)rr, pf = (float)q.rr_prev;
                        if (rf > FLT_MIN && pf > FLT_MIN && rf < FLT_MAX && pf < FLT_MAX) {
                            const float inv = 1.f / rf, b = rf / pf;
                            q.beta = (double)b;
                            q.c_re = (double)(1.f - b * ((float)s[2] * inv));
                            q.c_im = (double)(-b * ((float)s[3] * inv));
                        } else {
                            const double b = rr / q.rr_prev, inv = 1.0 / rr;
                            q.beta = b;
                            q.c_re = 1.0 - b * (s[2] * inv);
                            q.c_im = -b * (s[3] * inv);
                        }
                        q.mode = kSmRedo;
                        q.rmax2 = rr;
                    }
                    __syncwarp();
                    if (lane == 0) st = q;
                }
                __syncthreads();
                if (st.mode == kSmDone) break;
                beta = (W)st.beta;
                cre = (W)st.c_re;
                cim = (W)st.c_im;
            }
        }
        // ---------------- U: r and p (and x) of the next iteration
        if (st.mode == kSmStep) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = tid + u * TB;
                if (i < units) {
                    Un rv = sr[i + 2 * Nx], pv = sp[i + 2 * Nx];
#pragma unroll
                    for (int q = 0; q < 2 * K; ++q) {
                        rv.v[q] = fma(-alpha, ap[u].v[q], rv.v[q]);
                        x[u].v[q] = fma(alpha, pv.v[q], x[u].v[q]);
                        pv.v[q] = fma(beta, pv.v[q], rv.v[q]);
                    }
                    sr[i + 2 * Nx] = rv;
                    sp[i + 2 * Nx] = pv;
                }
                unit_end();
            }
            for (int h = tid; h < 4 * Nx; h += TB) {
                const int i = h < 2 * Nx ? h : h + units;
                const Un av = sa[h];
                Un rv = sr[i], pv = sp[i];
#pragma unroll
                for (int q = 0; q < 2 * K; ++q) {
                    rv.v[q] = fma(-alpha, av.v[q], rv.v[q]);
                    pv.v[q] = fma(beta, pv.v[q], rv.v[q]);
                }
                sr[i] = rv;
                sp[i] = pv;
            }
        } else {   // kSmRedo: p = c r + beta p
            for (int i = tid; i < units + 4 * Nx; i += TB) {
                const Un rv = sr[i];
                Un pv = sp[i];
#pragma unroll
                for (int q = 0; q < 2 * K; ++q) {
                    W c = cre * rv.v[q];
                    if constexpr (K == 2) c = fma(q & 1 ? cim : -cim, rv.v[q ^ 1], c);
                    pv.v[q] = fma(beta, pv.v[q], c);
                }
                sp[i] = pv;
            }
        }
        __syncthreads();
    }
    if constexpr (!MIXED) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = tid + u * TB;
            if (i < units) reinterpret_cast<Un*>(S.x)[2 * (size_t)n0 + i] = x[u];
        }
    }
    if (rank == 0 && tid == 0) {
        CGState& o = a.st[sys];
        o.rr = st.rr;
        o.rr0 = st.rr0;
        o.rr_prev = st.rr_prev;
        o.stop2 = st.stop2;
        o.rmax2 = st.rmax2;
        o.active = 0;
        o.iters = st.iters;
        o.converged = st.converged;
        o.status = st.status;
        o.n_ru = st.n_ru;
        o.mode = 0;
        o.chi_ready = st.ru;   // an update has just left D_first x of this x in t64
    }
    if (cluster_end(nc, &s_dead, &s_left, a.err) && rank == 0 && tid == 0) {
        CGState& o = a.st[sys];
        o.converged = 0;
        o.status = YK_ETIMEOUT;
    }
}

// Failure detection without a fault: four CTAs, of which CTA 1 waits for bytes that nobody
// sends, gives up and ends, while the others pass two more barriers, as in a reliable
// update, and then store into it.  out: the stores that CTA 1 found when all had
// come to the end, and the CTAs that learned of the timeout.
constexpr int kProbeCtas = 4;
__device__ int g_cluster_probe[3];   // err, out[2]

__global__ void __launch_bounds__(64) cluster_timeout_probe_kernel(int* err, int* out)
{
    __shared__ __align__(8) uint64_t mb[2];
    __shared__ __align__(8) double in[kProbeCtas];
    __shared__ int s_dead, s_left;
    unsigned rank;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const unsigned mb0 = (unsigned)__cvta_generic_to_shared(mb);
    if (threadIdx.x == 0) {
        s_dead = s_left = 0;
        for (int q = 0; q < kProbeCtas; ++q) in[q] = 0.0;
        for (int q = 0; q < 2; ++q) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb0 + 8u * q) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mb_expect(mb0, 16u);   // never sent
        mb_expect(mb0 + 8u, 8u * (kProbeCtas - 1));
    }
    __syncthreads();
    cluster_barrier();
    if (rank == 1) {
        mb_wait(mb0, 0, &s_dead);
    } else {
        cluster_barrier();
        cluster_barrier();
        if (threadIdx.x == 0) st_async(cta_addr(&in[rank], 1), 1.0, cta_addr(mb + 1, 1));
    }
    const bool late = cluster_end(kProbeCtas, &s_dead, &s_left, err);
    if (threadIdx.x == 0) {
        if (late) atomicAdd(out + 1, 1);
        if (rank == 1) {
            mb_wait(mb0 + 8u, 0, &s_dead);
            out[0] = (int)(in[0] + in[2] + in[3]);
        }
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {

struct SmForm {
    int c, threads, u;
    size_t smem;
};

size_t small_smem(int V, int Nx, int c, int K, bool mixed, bool pions)
{
    const size_t w = mixed ? 4 : 8, site = 4 * K * w, omax = (V + c - 1) / c;
    return (3 * (omax + 2 * Nx) + 2 * Nx) * site + omax * w * (pions ? 4 : 1);
}

const void* small_fn(int K, bool mixed, int u)
{
#define YK_SM(W, K_)                                                                                        \
    (u == 1 ? (const void*)cg_small_kernel<W, K_, 1> : u == 2 ? (const void*)cg_small_kernel<W, K_, 2>      \
     : (const void*)cg_small_kernel<W, K_, 4>)
    if (K == 1) return YK_SM(double, 1);   // at most 4 (kSmMaxReal)
    if (mixed) return u == 6 ? (const void*)cg_small_kernel<float, 2, 6> : YK_SM(float, 2);
    return YK_SM(double, 2);   // at most 4: its smaller shared memory holds no more
#undef YK_SM
}

// Opts every form in to its cluster size and shared memory; the largest
// cluster that can be resident (16, or 8 where a GPC holds no 16).
int small_max_cluster()
{
    return once_per_device([] {
        int best = 0;
        for (int K = 1; K <= 2; ++K)
            for (int m = 0; m <= (K == 2 ? 1 : 0); ++m)
                for (int u : {1, 2, 4, 6}) {
                    const void* fn = small_fn(K, m, u);
                    if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
                        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmMaxSmem) !=
                            cudaSuccess) {
                        cudaGetLastError();
                        return 0;
                    }
                    for (int c = kSmMaxC; c >= 8; c /= 2) {
                        cudaLaunchConfig_t cfg = {};
                        cfg.gridDim = dim3(c);
                        cfg.blockDim = dim3(kSmThreads);
                        cfg.dynamicSmemBytes = kSmMaxSmem;
                        cudaLaunchAttribute at[1];
                        at[0].id = cudaLaunchAttributeClusterDimension;
                        at[0].val.clusterDim.x = c;
                        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
                        cfg.attrs = at;
                        cfg.numAttrs = 1;
                        int n = 0;
                        if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
                            cudaGetLastError();
                            n = 0;
                        }
                        if (n >= 1) {
                            best = best == 0 ? c : (c < best ? c : best);
                            break;
                        }
                        if (c == 8) return 0;
                    }
                }
        return best;
    });
}

}  // namespace

// Whether the solve's systems, all on one lattice, take cg_small_kernel: its
// CTAs per system, threads and units a thread.  A real FP64 solve stays in the
// cluster up to 12288 sites (128 x 96: 19.5 us an iteration here, 23.5 in cg_kernel).
// The 16 SMs' FP64 pipes need as long as cg_kernel's synchronisations over the whole
// GPU a little above that: 112 x 112 20.7 against 23.8 us, 120 x 120 22.9 against 23.9,
// 128 x 128 25.3 against 23.7 (the line was drawn before the exchange by mbarriers; of
// several systems each has its own SMs here: four of 128 x 128 25.3 against 39.7).
// Complex solves stay while their vectors fit.
static bool small_form(const CGArgs& a, int K, bool mixed, const OneLattice& lat, SmForm* f)
{
    const int Nt = lat.Nt, Nx = lat.Nx;
    if (Nt < 2 || Nx < 2 || a.balance != nullptr || (K == 1 && mixed)) return false;
    const int V = Nt * Nx;
    if (K == 1 && V > kSmMaxReal) return false;
    int c = small_max_cluster();
    if (c == 0) return false;
    // a CTA owns at least a row (its neighbours hold all that surrounds it)
    while (c > Nt) c /= 2;
    auto fits = [&](int q) {
        const int u = (2 * ((V + q - 1) / q) + kSmThreads - 1) / kSmThreads;
        return u <= (mixed ? 6 : 4) && small_smem(V, Nx, q, K, mixed, lat.pions != 0) <= kSmMaxSmem;
    };
    if (!fits(c)) return false;
    // 32 sites a CTA at least, and up to 288 CTAs in all: 18 clusters of 16, as many as are
    // resident at two such CTAs an SM (us an iteration, 32 x 32, 18 systems on 16 CTAs each
    // 6.4, on 8 7.6; 36 on 8 7.9, on 16 12.2; 64 x 64, 18 on 16 24.0, on 8 27.1).  It is not
    // the best for every count: 54 x 45, 24 systems on 8 18.1, on 4 16.1; 32 x 32, 19 on 8
    // 7.6, on 16 6.5.
    while (c > 1 && (V / c < 32 || (long long)c * a.sys_count > 288) && fits(c / 2)) c /= 2;
    const int units = 2 * ((V + c - 1) / c);
    int u = 1;
    while (u * kSmThreads < units) u = u == 4 ? 6 : 2 * u;
    f->c = c;
    f->u = u;
    f->threads = ((units + u - 1) / u + 31) / 32 * 32;
    f->smem = small_smem(V, Nx, c, K, mixed, lat.pions != 0);
    return true;
}

void cg_small_init() { small_max_cluster(); }

int cg_small_grid(const CGArgs& a, int K, bool mixed, const OneLattice& lat)
{
    SmForm f;
    return small_form(a, K, mixed, lat, &f) ? f.c * a.sys_count : 0;
}

cudaError_t launch_cg_small(const CGArgs& a, int K, bool mixed, const OneLattice& lat, cudaStream_t stream)
{
    SmForm f;
    if (!small_form(a, K, mixed, lat, &f)) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(f.c * a.sys_count);
    cfg.blockDim = dim3(f.threads);
    cfg.dynamicSmemBytes = f.smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = f.c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CGArgs b = a;
    int pions = lat.pions;
    void* args[] = {&b, &pions};
    return cudaLaunchKernelExC(&cfg, small_fn(K, mixed, f.u), args);
}

int cluster_timeout_probe(cudaStream_t stream, int* status)
{
    void* p = nullptr;
    int h[3] = {};
    cudaError_t e = cudaGetSymbolAddress(&p, g_cluster_probe);
    if (e == cudaSuccess) e = cudaMemsetAsync(p, 0, sizeof(h), stream);
    if (e == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kProbeCtas);
        cfg.blockDim = dim3(64);
        cfg.stream = stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kProbeCtas;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int *err = (int*)p, *out = err + 1;
        void* args[] = {&err, &out};
        e = cudaLaunchKernelExC(&cfg, (const void*)cluster_timeout_probe_kernel, args);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, p, sizeof(h), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return -1;
    *status = h[1] == kProbeCtas - 1 && h[2] == kProbeCtas ? h[0] : 0;
    return 0;
}

}  // namespace yk

// yk_cg_eoc.cu -- the step's even-odd solve (the Schur-complement CGNE of
// cg_eo_kernel, yk_cg.cu: its equations, stopping rule and reliable updates)
// inside one thread-block cluster per system, for lattices whose vectors fit
// the registers and shared memory of at most 16 SMs (256 x 256 and smaller).
//
// What bounds these solves is latency and L2 traffic: cg_eo_kernel spends a
// grid barrier and the staging of three widened vectors per iteration, the
// batched kernels (cg_eop_kernel, cg_eob_kernel) deal every patch of every
// system out again in every round.  Here a CTA owns rows of the compact lattice
// for the whole solve and nothing but the two edge rows of v and q and four
// sums leaves it in an iteration:
//   w = -A_o^-1 H_oe p      on the own rows and one around them
//   v = A_e p + H_eo w      on the own rows; its edge rows also go into the
//                           neighbours' shared memory       -> their threads at the edges
//   u = -A_o^-1 H^dag_oe v  on the own rows and one around them
//   q = A_e v + H^dag_eo u  on the own rows; edge rows into the neighbours, the
//                           sums' partials into every CTA   -> the scalar step, then q's rows
//   chi_e += alpha v, r -= alpha q, p = r + beta p on the own rows; r and p also
//                           on the two rows around them, from the neighbours' q
// What leaves is stored asynchronously and counted on the receiver's mbarriers, and only those
// threads wait that read it; there is no cluster barrier but in an update.
// Systems run independently: no block waits for another system's.
//
// A thread owns up to U consecutive rows of one compact column, and the chi
// increment, r, p, v, and w, u and q of its sites stay in its registers.  An
// even-odd hop has one of its two x neighbours at the site's own compact index
// and its time neighbours a row up and down, so from shared memory it takes only
// the other x neighbour and, at the ends of a thread's rows, the next threads'
// rows; at r = 1 the neighbour stores of these only what its hop keeps (one spin
// combination, one spin entry: 8 bytes of 16), and a hop takes 8 operations per
// spin pair against 14.  Rows carry no case distinctions: the x neighbours' offsets
// and signs alternate from row to row, and a value that crosses the antiperiodic
// boundary is stored into the rows around a CTA's own with its sign changed.
#include <cfloat>
#include <type_traits>

#include "yk_cluster.cuh"
#include "yk_kernels.h"

namespace yk {

namespace {

constexpr int kEcMaxC = 16;
constexpr int kEcThreads = 512;
constexpr int kEcMaxU = 4;

enum EcMode { kEcStep = 1, kEcRu = 2, kEcRedo = 3, kEcDone = 4 };

// The solve's scalar state, written by thread 0, the same bits in every CTA: what
// the passes read, then what only the scalar steps use.
struct EcState {
    float alpha, beta, c_re;
    int mode, ru;   // ru: an update has just formed the odd hop of the present chi_e
    float stop2f, rmax2, rr_prev, delta2;
    int due, n_ru, iters, converged, status;
    float est, rr_min;   // the recursion's |r|^2 where it asked for an update (0: it met the target); the lowest found
    int stray;           // the first update since whose residual did not follow it (-1: none)
    double stop2, rr_ref, rr;
};

// Whether float-float's residual, rf after the update of iteration k, has reached its floor
// above the target: it no longer falls by a factor (4 in the square), though the recursion does, for a
// sixteenth of the iterations so far and eight (a solve that is near the floor may still get
// through in that time).  For solves with another to fall back on.
__device__ __forceinline__ bool falls_no_further(EcState& st, int k, float rf)
{
    if (rf <= 0.25f * st.rr_min) {
        st.rr_min = rf;
        st.stray = -1;
    } else if (st.stray < 0 && rf > 4.f * st.est) {
        st.stray = k;
    }
    return st.stray >= 0 && k - st.stray >= st.stray / 16 + 8;
}

__device__ __forceinline__ float4 f4_zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }

__device__ __forceinline__ float4 f4_mul(float a, float4 x) { return make_float4(a * x.x, a * x.y, a * x.z, a * x.w); }

__device__ __forceinline__ float4 f4_fma(float a, float4 x, float4 y)
{
    return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}

__device__ __forceinline__ float f4_dot(float4 a, float4 b, float s)
{
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}

// A store at such an address of another CTA.
__device__ __forceinline__ void st_cta(unsigned addr, float4 v)
{
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

// What a hop takes of a neighbour: at r = 1 two numbers (one for each flavour),
// else the site.
template <bool R1>
struct Part {
    using T = float2;
};
template <>
struct Part<false> {
    using T = float4;
};

// of the x neighbour with another compact index, e the hop's sign (below)
template <bool R1>
__device__ __forceinline__ typename Part<R1>::T part_x(float4 s, float e)
{
    if constexpr (R1)
        return make_float2(fmaf(e, s.y, s.x), fmaf(e, s.w, s.z));
    else
        return s;
}

// of the neighbour at t + 1 (UP) or t - 1: D keeps spin d of the first, u of the second
template <bool DAG, bool UP, bool R1>
__device__ __forceinline__ typename Part<R1>::T part_t(float4 s)
{
    if constexpr (R1)
        return DAG == UP ? make_float2(s.x, s.z) : make_float2(s.y, s.w);
    else
        return s;
}

// v, whose later uses the compiler does not merge with others
__device__ __forceinline__ int opaque(int v)
{
    asm volatile("" : "+r"(v));
    return v;
}

// diag c + H of one site (C; else H alone; D; DAG: D^dag) from its neighbours'
// parts, dn (t - 1), up (t + 1) and oth, and the x neighbour `same` at its own
// compact index.  e: +1 where D (DAG: -1) and `same` is the upper x neighbour.
template <bool DAG, bool C, bool R1, typename T = typename Part<R1>::T>
__device__ __forceinline__ float4 hop(float4 c, float diag, T dn, float4 same, T up, T oth, float e, float r)
{
    float4 o;
    const float h = 0.5f * e;
    if constexpr (R1) {
        const float a0 = fmaf(-e, same.y, same.x), a1 = fmaf(-e, same.w, same.z);
        const T u = DAG ? up : dn, d = DAG ? dn : up;
        auto site = [&](float cv, float t) { return C ? fmaf(diag, cv, -t) : -t; };
        o.x = fmaf(-0.5f, a0 + oth.x, site(c.x, u.x));
        o.y = fmaf(h, a0 - oth.x, site(c.y, d.x));
        o.z = fmaf(-0.5f, a1 + oth.y, site(c.z, u.y));
        o.w = fmaf(h, a1 - oth.y, site(c.w, d.y));
    } else {
        const float P = -0.5f * (r + 1.f), M = -0.5f * (r - 1.f), A = -0.5f * r;
        const float uu = DAG ? P : M, ud = DAG ? M : P;   // of t + 1; t - 1 takes them exchanged
        auto site = [&](float cv, float t) { return C ? fmaf(diag, cv, t) : t; };
        o.x = fmaf(ud, dn.x, site(c.x, uu * up.x));
        o.y = fmaf(uu, dn.y, site(c.y, ud * up.y));
        o.z = fmaf(ud, dn.z, site(c.z, uu * up.z));
        o.w = fmaf(uu, dn.w, site(c.w, ud * up.w));
        o.x = fmaf(A, same.x + oth.x, fmaf(h, same.y - oth.y, o.x));
        o.y = fmaf(A, same.y + oth.y, fmaf(h, same.x - oth.x, o.y));
        o.z = fmaf(A, same.z + oth.z, fmaf(h, same.w - oth.w, o.z));
        o.w = fmaf(A, same.w + oth.w, fmaf(h, same.z - oth.z, o.w));
    }
    return o;
}

__device__ __forceinline__ SiteFF ff_join(float4 h, float4 l)
{
    return SiteFF{{FF{h.x, l.x}, FF{h.y, l.y}, FF{h.z, l.z}, FF{h.w, l.w}}};
}

__device__ __forceinline__ float4 ff_hi(const SiteFF& s) { return make_float4(s.v[0].hi, s.v[1].hi, s.v[2].hi, s.v[3].hi); }
__device__ __forceinline__ float4 ff_lo(const SiteFF& s) { return make_float4(s.v[0].lo, s.v[1].lo, s.v[2].lo, s.v[3].lo); }

// H^dag in float-float.
template <bool R1>
__device__ __forceinline__ SiteFF hop_dag_ff(const SiteFF& dn, const SiteFF& same, const SiteFF& up, const SiteFF& oth,
                                             float sg, FF r)
{
    SiteFF o;
    if constexpr (R1) {
        const float h = -0.5f * sg;
#pragma unroll
        for (int f = 0; f < 4; f += 2) {
            const FF a = ff_add(same.v[f], ff_sign(same.v[f + 1], sg));
            const FF b = ff_add(oth.v[f], ff_sign(oth.v[f + 1], -sg));
            const FF s = ff_add(a, b), d = ff_sub(a, b);
            o.v[f] = ff_sub(FF{-0.5f * s.hi, -0.5f * s.lo}, up.v[f]);
            o.v[f + 1] = ff_sub(FF{h * d.hi, h * d.lo}, dn.v[f + 1]);
        }
    } else {
        const FF rp = ff_add(r, FF{1.f, 0.f}), rm = ff_add(r, FF{-1.f, 0.f});
        const FF P = ff_sign(rp, -0.5f), M = ff_sign(rm, -0.5f), A = ff_sign(r, -0.5f);
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const int g = f ^ 1;   // spin u: P of t + 1, M of t - 1; spin d exchanged
            FF t = ff_add(ff_mul(f & 1 ? M : P, up.v[f]), ff_mul(f & 1 ? P : M, dn.v[f]));
            t = ff_add(t, ff_sign(ff_sub(same.v[g], oth.v[g]), -0.5f * sg));
            o.v[f] = ff_add(t, ff_mul(A, ff_add(same.v[f], oth.v[f])));
        }
    }
    return o;
}

// A CTA's share of a system and its buffers (below).
struct EcView {
    int Nh, r0, rows, at_prv, at_nxt;
    unsigned to_prv, to_nxt;
    float f_prv, f_nxt;
    double *chi, *rhs;
    float4 *base, *P, *L, *V, *W, *RH, *QH, *p_own;   // p_own: global memory, p of the own rows
    float *deh, *del, *dih, *dil;

    // an edge row's value into the neighbours' copies of it: cell j of a buffer is
    // the previous CTA's cell j + its rows, the next one's cell j - rows; in the
    // four-row halos of RH and QH cells j and j - rows
    __device__ __forceinline__ void send(const float4* buf, bool halo, bool to_p, bool to_n, int j, float4 v) const
    {
        const int b = (int)(buf - base) + j;
        if (to_p) st_cta(to_prv + 16u * (unsigned)(b + (halo ? 0 : at_prv)), f4_mul(f_prv, v));
        if (to_n) st_cta(to_nxt + 16u * (unsigned)(b + at_nxt), f4_mul(f_nxt, v));
    }
};

// A reliable update in float-float, the increment x in W, v in V and p in p_own:
// chi_e += x + al v (its parts with two rows around into V and W); the odd hop
// -A_o^-1 H^dag_oe chi_e into P and L; then, unless only_odd, r = rhs_e - (A_e chi_e +
// H^dag_eo of it), in FP32, into V and its edge rows into the neighbours' RH.
// Returns the thread's |r|^2 and <r, p>, float-float.  Out of line: the
// iterations' registers need not hold through it.
template <bool R1>
__device__ __noinline__ float4 ec_update(const EcView& g, float al, bool only_odd, FF rr)
{
    const int Nh = g.Nh, rows = g.rows, NS = kEcThreads / Nh;
    const int strip = threadIdx.x / Nh, i = threadIdx.x - strip * Nh;
    const int per = (rows + NS - 1) / NS, perw = (rows + 2 + NS - 1) / NS;
    const int o0 = strip * per, o1 = strip < NS ? min(o0 + per, rows) : o0;
    const int w0 = strip * perw - 1, w1 = strip < NS ? min(w0 + perw, rows + 1) : w0;
    const int up_x = i + 1 == Nh ? 1 - Nh : 1, dn_x = i == 0 ? Nh - 1 : -1;
    const int m0 = g.r0 * Nh + i, j0 = 2 * Nh + i;   // of row 0
    SiteFF ahead = {};   // what the next row takes from global memory, a row ahead
    if (o0 < o1) ahead = ld_ff(g.chi, m0 + o0 * Nh);
#pragma unroll 1
    for (int row = o0; row < o1; ++row) {
        const int j = j0 + row * Nh, m = m0 + row * Nh;
        SiteFF c = ahead;
        if (row + 1 < o1) ahead = ld_ff(g.chi, m + Nh);
        const float4 v4 = g.V[j], x4 = g.W[j];
        const float vv[4] = {v4.x, v4.y, v4.z, v4.w}, xv[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float pr = __fmul_rn(al, vv[e]);   // alpha v exactly: (pr, its FMA error)
            c.v[e] = ff_add(c.v[e], FF{xv[e], 0.f});
            c.v[e] = ff_add(c.v[e], FF{pr, __fmaf_rn(al, vv[e], -pr)});
        }
        st_ff(g.chi, m, c);
        const float4 hi = ff_hi(c), lo = ff_lo(c);
        g.V[j] = hi;
        g.W[j] = lo;
        g.send(g.V, false, row < 2, row >= rows - 2, j, hi);
        g.send(g.W, false, row < 2, row >= rows - 2, j, lo);
    }
    float4 pn = f4_zero();
    if (o0 < o1) {
        ahead = ld_ff(g.rhs, m0 + o0 * Nh);
        pn = g.p_own[m0 + o0 * Nh];
    }
    cluster_barrier();
    FF s0 = {0.f, 0.f}, s2 = {0.f, 0.f};
    // the odd sites, then the even ones
#pragma unroll 1
    for (int odd = 1; odd >= (only_odd ? 1 : 0); --odd) {
        const float4 *hi = odd ? g.V : g.P, *lo = odd ? g.W : g.L;
        const int end = odd ? w1 : o1;
#pragma unroll 1
        for (int row = odd ? w0 : o0; row < end; ++row) {
            const int j = j0 + row * Nh;
            const bool b = (g.r0 + row + odd) & 1;
            const int jo = j + (b ? up_x : dn_x);
            SiteFF h = hop_dag_ff<R1>(ff_join(hi[j - Nh], lo[j - Nh]), ff_join(hi[j], lo[j]),
                                      ff_join(hi[j + Nh], lo[j + Nh]), ff_join(hi[jo], lo[jo]), b ? -1.f : 1.f, rr);
            if (odd) {
                const FF inv = {-g.dih[j - Nh], -g.dil[j - Nh]};
#pragma unroll
                for (int c = 0; c < 4; ++c) h.v[c] = ff_mul(inv, h.v[c]);
                g.P[j] = ff_hi(h);
                g.L[j] = ff_lo(h);
            } else {
                const SiteFF b4 = ahead, c4 = ff_join(g.V[j], g.W[j]);
                const float4 p = pn;
                if (row + 1 < o1) {
                    ahead = ld_ff(g.rhs, m0 + (row + 1) * Nh);
                    pn = g.p_own[m0 + (row + 1) * Nh];
                }
                const FF de = {-g.deh[j - 2 * Nh], -g.del[j - 2 * Nh]};
#pragma unroll
                for (int c = 0; c < 4; ++c) h.v[c] = ff_add(b4.v[c], ff_sub(ff_mul(de, c4.v[c]), h.v[c]));
                const float4 r4 = ff_hi(h);
                g.V[j] = r4;   // chi_e's high parts have had their last use by others
                g.send(g.RH, true, row < 2, row >= rows - 2, j, r4);
                s0 = ff_add(s0, FF{f4_dot(r4, r4, 0.f), 0.f});
                s2 = ff_add(s2, FF{f4_dot(r4, p, 0.f), 0.f});
            }
        }
        __syncthreads();
    }
    return make_float4(s0.hi, s0.lo, s2.hi, s2.lo);
}

}  // namespace

// What a solve starts from, at every compact site of the tiles' systems: the
// sources (kept in b for the force), A_e (v32) and 1 / A_o (dinv) in float-float,
// chi_e = 0, rhs_e = eta_e - H^dag_eo A_o^-1 eta_o, and the tile's |eta|^2
// (its partial's first slot).  A kernel of its own because it has the whole GPU:
// inside the solve it took 26 of 195 us at 256 x 256, on 16 SMs.  A block forms
// -A_o^-1 eta_o on its tile and a row around it in shared memory.  err, when given, is
// cleared: here, before all solves of the step, since one that starts late would clear
// what another has recorded.
template <bool R1>
__global__ void __launch_bounds__(kTile) eoc_prepare_kernel(CGArgs a, int* err)
{
    extern __shared__ __align__(16) float4 ep_raw[];   // high parts, then low
    __shared__ FF red[kTile / 32];
    if (err && blockIdx.x == 0 && threadIdx.x == 0) *err = 0;
    const int idx = a.tile_begin + (int)blockIdx.x;
    const int2 tl = a.eo_tiles[idx];
    const SysDev& S = a.sys[tl.x];         // the compact view
    const SysDev& SF = a.sys_full[tl.x];   // the full record
    if (idx < S.tile0 || idx >= S.tile0 + S.ntiles) return;   // the full table has more tiles
    if (R1 != (S.r == 1.0)) return;
    const int Nh = S.Nx, Ve = S.V, m0 = tl.y;
    float4* const hi = ep_raw;
    float4* const lo = ep_raw + kTile + 2 * Nh;
    const bool gen = SF.gen_eta != 0;   // generated sources are FP32 normals
    const int64_t step = gen ? *SF.step : 0;
    const double* const ahead = gen && a.eta_kind == 2 && SF.eta_tag && SF.eta_tag[step & 1] == step
                                    ? SF.eta_ahead[step & 1] : nullptr;
    const double diag0 = 2.0 * S.r + S.m0;
    FF eta2 = {0.f, 0.f};
    // the odd sites of the tile and around it, then the tile's even ones
    const int odds = min(kTile, Ve - m0) + 2 * Nh;
    const int np = (odds + kTile - 1) / kTile;
#pragma unroll 1
    for (int pass = 0; pass <= np; ++pass) {
        const bool odd = pass < np;
        if (!odd) __syncthreads();
        const int c = threadIdx.x + (odd ? pass * kTile : Nh);
        int m = m0 - Nh + c;
        const bool across = m < 0 || m >= Ve, own = c >= Nh && c < odds - Nh;
        if (odd ? c >= odds : !own) continue;
        m = m < 0 ? m + Ve : (m >= Ve ? m - Ve : m);
        const int t = m / Nh, i = m - t * Nh;
        const bool b = (t + (odd ? 1 : 0)) & 1;
        const int n = 2 * m + (b ? 1 : 0);
        const FF d = ff_split(fma((double)S.g, SF.sigma[n], diag0));
        SiteFF e;
        if (gen && !ahead) {
            e = ff_join(normal4(rng_stream(SF.seed, (uint32_t)SF.chain, (uint64_t)step, (uint32_t)a.eta_kind,
                                           (uint32_t)SF.rhs), (uint32_t)n), f4_zero());
        } else {
            const Site<double, 1> q = load_site<double, 1>(gen ? ahead : SF.b, n);
#pragma unroll
            for (int k = 0; k < 4; ++k) e.v[k] = gen ? FF{narrow(q.v[k]), 0.f} : ff_split(q.v[k]);
        }
        if (own) {
            if (gen) {
                Site<double, 1> q;
#pragma unroll
                for (int k = 0; k < 4; ++k) q.v[k] = widen(e.v[k].hi);
                store_site<double, 1>(SF.b, n, q);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) eta2 = ff_add(eta2, ff_mul(e.v[k], e.v[k]));
        }
        if (odd) {
            FF inv = ff_rcp(d);
            if (own) st_ff1(S.dinv, m, inv);
            inv = ff_sign(inv, across ? 1.f : -1.f);
#pragma unroll
            for (int k = 0; k < 4; ++k) e.v[k] = ff_mul(inv, e.v[k]);
            hi[c] = ff_hi(e);
            lo[c] = ff_lo(e);
        } else {
            const int co = c + (b ? (i + 1 == Nh ? 1 - Nh : 1) : (i == 0 ? Nh - 1 : -1));
            SiteFF h = hop_dag_ff<R1>(ff_join(hi[c - Nh], lo[c - Nh]), ff_join(hi[c], lo[c]),
                                      ff_join(hi[c + Nh], lo[c + Nh]), ff_join(hi[co], lo[co]), b ? -1.f : 1.f,
                                      R1 ? FF{1.f, 0.f} : ff_of(S.r));
#pragma unroll
            for (int k = 0; k < 4; ++k) h.v[k] = ff_add(h.v[k], e.v[k]);
            st_ff(S.x, m, SiteFF{});
            st_ff(S.x, Ve + m, h);
            st_ff1(reinterpret_cast<double*>(S.v32), m, d);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) eta2 = ff_add(eta2, ff_shfl_xor(eta2, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = eta2;
    __syncthreads();
    if (threadIdx.x == 0) {
        FF q = red[0];
        for (int w = 1; w < kTile / 32; ++w) q = ff_add(q, red[w]);
        a.partial[idx].f[0] = make_float2(q.hi, q.lo);
    }
}

// FULL: every thread that owns rows owns U of them.
template <int U, bool FULL, bool R1>
__global__ void __launch_bounds__(kEcThreads, 1) cg_eoc_kernel(CGArgs a, const int* __restrict__ order, int cells, int first_cells)
{
    extern __shared__ __align__(16) float4 ec_raw[];
    __shared__ FF wred[kEcThreads / 32][4];
    __shared__ __align__(8) FF cpart[2][kEcMaxC][4];   // by the iteration's parity
    __shared__ __align__(8) uint64_t mb[4];   // arrivals: VH, QH, cpart[0], cpart[1]
    __shared__ int s_dead, s_left;
    __shared__ EcState st;
    __shared__ SysDev S;     // the compact view
    __shared__ EcView g;
    unsigned rank, nc;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(nc));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    {
        const int slot = (int)(blockIdx.x / nc);
        const int sys = order ? order[slot] : a.sys_first + slot;
        static_assert(sizeof(SysDev) % 8 == 0 && sizeof(SysDev) / 8 <= kEcThreads, "the records' copy");
        constexpr int n = sizeof(SysDev) / 8;
        if (tid < n) reinterpret_cast<uint64_t*>(&S)[tid] = reinterpret_cast<const uint64_t*>(a.sys + sys)[tid];
        if (tid == 0) {
            st.iters = sys;   // for the end: where the state goes
            s_dead = s_left = 0;
            for (int q = 0; q < 4; ++q)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(mb + q)));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    __syncthreads();
    CGState* const out_state = a.st + st.iters;
    const int Nt = S.Nt, Nh = S.Nx;
    const int r0 = (int)((unsigned)Nt * rank / nc), rows = (int)((unsigned)Nt * (rank + 1) / nc) - r0;
    // Buffers hold the CTA's rows and two around them on either side: row t of
    // [r0 - 2, r0 + rows + 2) is row t - r0, cell (row + 2) Nh + column.  The rows
    // around that lie across the lattice's time boundary hold the values' negatives.
    const int NB = cells;            // of a buffer, the same in every CTA
    const int DN = NB - 4 * Nh;
    // Round 0 and the updates use P, L (the parts of the odd hop) and V, W (of
    // chi_e); the iterations, in the place of P and L, the halos PH, VH, the parts
    // that hops take of the even (0) and odd (1) sites -- X of every own site, U
    // and D of the first and last row of every thread -- and A_e and 1 / A_o in
    // FP32 (DE, DI).  These are laid out by thread (row u of thread tid: u kEcThreads + tid),
    // so that every address is a thread's register and a constant.
    using E = typename Part<R1>::T;
    constexpr int kN = kEcThreads;
    const int NS = kN / Nh;
    float4* const P = ec_raw;
    float4* const L = P + NB;
    float4* const PH = ec_raw;       // p on the two rows before, then the two after
    float4* const VH = PH + 4 * Nh;  // v there
    E* const X0 = reinterpret_cast<E*>(VH + 4 * Nh);
    E* const X1 = X0 + U * kN;
    E* const U0 = X1 + U * kN;
    E* const D0 = U0 + kN;
    E* const U1 = D0 + kN;
    E* const D1 = U1 + kN;
    float* const DE = reinterpret_cast<float*>(D1 + kN);
    float* const DI = DE + U * kN;
    float4* const V = ec_raw + first_cells;
    float4* const W = V + NB;
    float4* const RH = W + NB;       // r on the rows around
    float4* const QH = RH + 4 * Nh;  // q there; in an update p
    float* const deh = reinterpret_cast<float*>(QH + 4 * Nh);   // A_e on the own rows
    float* const del = deh + DN;
    float* const dih = del + DN;     // 1 / A_o on the own rows and one around them (from row -1)
    float* const dil = dih + DN + 2 * Nh;

    // the thread's column and its strip of rows: own rows [o0, o0 + on); fs, ls: its
    // first, last is the CTA's
    const int strip = tid / Nh, i = tid - strip * Nh;
    const int per = (rows + NS - 1) / NS;
    const int o0 = strip * per, on = strip < NS ? max(min(per, rows - o0), 0) : 0;
    auto has = [&](int u) { return FULL || u < on; };        // among threads with on > 0
    auto last = [&](int u) { return FULL ? u + 1 == U : u + 1 == on; };
    const bool fs = on > 0 && o0 == 0, ls = on > 0 && o0 + on == rows;
    // the x neighbour with another compact index, relative to the cell: for a hop
    // to an even site xe in the thread's first row and every second after it, xe1
    // in the others; to an odd site exchanged; se: the hops' e of D to the even
    // sites in the first row
    const int up_x = i + 1 == Nh ? 1 - Nh : 1, dn_x = i == 0 ? Nh - 1 : -1;
    const bool eb = (r0 + o0) & 1;
    const int xe = eb ? up_x : dn_x, xe1 = eb ? dn_x : up_x;
    const float se = eb ? -1.f : 1.f;
    const int je = (o0 + 2) * Nh + i;   // the first own cell of a buffer
    const int te = tid + xe, te1 = tid + xe1;
    float rw = 1.f;
    FF rff = {1.f, 0.f};
    if constexpr (!R1) {
        rw = (float)S.r;
        rff = ff_of(S.r);
    }
    const unsigned nxt = rank + 1 == nc ? 0 : rank + 1, prv = rank == 0 ? nc - 1 : rank - 1;
    if (tid == 0) {
        const int prev_rows = (int)((unsigned)Nt * (prv + 1) / nc) - (int)((unsigned)Nt * prv / nc);
        double* const rhs = S.x + 4 * (size_t)S.V;   // after chi_e
        g = EcView{Nh, r0, rows, prev_rows * Nh, -rows * Nh, cta_addr(ec_raw, prv), cta_addr(ec_raw, nxt),
                   rank == 0 ? -1.f : 1.f, rank + 1 == nc ? -1.f : 1.f, S.x, rhs, ec_raw, P, L, V, W, RH, QH,
                   reinterpret_cast<float4*>(S.p32[0]), deh, del, dih, dil};
    }
    // row u's value of the thread, when it is an edge row, into the neighbours' halo
    const unsigned to_prv = cta_addr(ec_raw, prv) + 16u * (unsigned)je, to_nxt = cta_addr(ec_raw, nxt) + 16u * (unsigned)(je - rows * Nh);
    const float f_prv = rank == 0 ? -1.f : 1.f, f_nxt = rank + 1 == nc ? -1.f : 1.f;
    const unsigned mb0 = (unsigned)__cvta_generic_to_shared(mb);
    auto send_halo = [&](const float4* halo, int mbar, int u, bool to_p, bool to_n, float4 v) {
        const unsigned o = 16u * (unsigned)((int)(halo - ec_raw) + u * Nh);
        if (to_p) st_async(to_prv + o, f4_mul(f_prv, v), cta_addr(mb + mbar, prv));
        if (to_n) st_async(to_nxt + o, f4_mul(f_nxt, v), cta_addr(mb + mbar, nxt));
    };
    // whether row u of the thread is among the CTA's first (last) two
    const bool first2 = U == 1 ? on > 0 && o0 < 2 : fs, last2 = U == 1 ? on > 0 && o0 >= rows - 2 : ls;
    auto edge_p = [&](int u) { return FULL ? (u < 2 && first2) : o0 + u < 2; };
    auto edge_n = [&](int u) { return FULL ? (u >= U - 2 && last2) : o0 + u >= rows - 2; };
    // (What only the CTA's edge rows need is read again where it is used: held in
    // registers through the iterations it spilled others.)
    // w = -A_o^-1 H f (DAG: H^dag) at the thread's sites from f, its parts in X0, U0, D0
    // and its halo H; lo, hi: the parts that the next hops take of the CTA's rows
    // -1 and `rows`
    auto odd_pass = [&](auto dag, const float4 (&f)[U], const float4* H, float4 (&w)[U], E& lo, E& hi) {
        constexpr bool DAG = decltype(dag)::value;
        if (on == 0) return;
        const float e0 = DAG ? se : -se;   // of the first row, the hop to an odd site
        E dn, end;
        if (fs) {   // row -1: as the even sites of row 0
            const float4* const h0 = H + opaque(i);
            const int nh = *(const volatile int*)&g.Nh;
            dn = part_t<DAG, false, R1>(h0[nh]);
            const float4 h = hop<DAG, false, R1>(f4_zero(), 0.f, part_t<DAG, false, R1>(h0[0]), h0[nh],
                                                 part_t<DAG, true, R1>(f[0]), part_x<R1>(h0[nh + xe], -e0), -e0, rw);
            lo = part_t<DAG, false, R1>(f4_mul(-dih[opaque(i)], h));
        } else {
            dn = D0[tid - Nh];
        }
        if (ls)
            end = part_t<DAG, true, R1>(H[2 * *(const volatile int*)&g.Nh + i]);
        else
            end = U0[tid + Nh];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (has(u)) {
                const float e = u & 1 ? -e0 : e0;
                const E up = last(u) ? end : part_t<DAG, true, R1>(f[u + 1 < U ? u + 1 : u]);
                const float4 h = hop<DAG, false, R1>(f4_zero(), 0.f, dn, f[u], up, X0[u * kN + (u & 1 ? te : te1)], e, rw);
                w[u] = f4_mul(-DI[u * kN + tid], h);
                dn = part_t<DAG, false, R1>(f[u]);
                X1[u * kN + tid] = part_x<R1>(w[u], -e);   // for the hop to the even sites
                if (u == 0) U1[tid] = part_t<DAG, true, R1>(w[0]);
                if (last(u)) D1[tid] = part_t<DAG, false, R1>(w[u]);
            }
        if (ls) {   // row `rows`: the next row after the thread's last, on - 1
            const bool odd = (FULL ? U : on) & 1;
            const float e = odd ? -e0 : e0;
            const int nh = *(const volatile int*)&g.Nh;
            const float4* const h2 = H + 2 * nh + i;
            const float4 h = hop<DAG, false, R1>(f4_zero(), 0.f, dn, h2[0], part_t<DAG, true, R1>(h2[nh]),
                                                 part_x<R1>(h2[odd ? xe : xe1], e), e, rw);
            hi = part_t<DAG, true, R1>(f4_mul(-dih[(*(const volatile int*)&g.rows + 1) * nh + i], h));
        }
    };
    // A_e c + H w (DAG: H^dag) at the thread's sites, w's parts in X1, U1, D1:
    // f(u, row, value), after which w[u] may change
    auto even_pass = [&](auto dag, const float4 (&c)[U], const float4 (&w)[U], E lo, E hi, auto&& f) {
        constexpr bool DAG = decltype(dag)::value;
        if (on == 0) return;
        const float e0 = DAG ? -se : se;
        E dn = fs ? lo : D1[tid - Nh];
        const E end = ls ? hi : U1[tid + Nh];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (has(u)) {
                const E up = last(u) ? end : part_t<DAG, true, R1>(w[u + 1 < U ? u + 1 : u]);
                const float4 h = hop<DAG, true, R1>(c[u], DE[u * kN + tid], dn, w[u], up, X1[u * kN + (u & 1 ? te1 : te)],
                                                    u & 1 ? -e0 : e0, rw);
                dn = part_t<DAG, false, R1>(w[u]);
                f(u, h);
            }
    };
    // the parts of an even vector that the hops (DAG: H^dag) to the odd sites take
    auto publish = [&](auto dag, int u, float4 f) {
        constexpr bool DAG = decltype(dag)::value;
        const float e = (u & 1) != DAG ? se : -se;
        X0[u * kN + tid] = part_x<R1>(f, e);
        if (u == 0) U0[tid] = part_t<DAG, true, R1>(f);
        if (last(u)) D0[tid] = part_t<DAG, false, R1>(f);
    };
    // A_e and 1 / A_o of the thread's sites for the iterations
    auto diagonals = [&] {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < on) {
                DE[u * kN + tid] = deh[(o0 + u) * Nh + i];
                DI[u * kN + tid] = dih[(o0 + u + 1) * Nh + i];
            }
    };
    // the CTA's four sums into every CTA's cpart
    auto partials = [&](const auto& v, int b, bool async) {
        const auto c = warp_sum4(v);
        if ((lane & 7) == 0) wred[warp][lane >> 3] = s_of(c, FF{});
        __syncthreads();
        if (warp == 0) {
            const int v4 = lane >> 3, q = lane & 7;
            FF t = ff_add(wred[q][v4], wred[q + 8][v4]);
            t = ff_add(t, ff_shfl_xor(t, 4));
            t = ff_add(t, ff_shfl_xor(t, 2));
            t = ff_add(t, ff_shfl_xor(t, 1));
            for (unsigned c2 = q; c2 < nc; c2 += 8)
                if (async)
                    st_async(cta_addr(&cpart[b][rank][v4], c2), t, cta_addr(mb + 2 + b, c2));
                else
                    *in_cta(&cpart[b][rank][v4], c2) = t;
        }
    };
    // the cluster's sums, in every lane of warp 0
    auto totals = [&](FF (&s)[4], int b) {
        const int v4 = lane >> 3, q = lane & 7;
        FF t = q < (int)nc ? cpart[b][q][v4] : FF{0.f, 0.f};
        if (q + 8 < (int)nc) t = ff_add(t, cpart[b][q + 8][v4]);
        t = ff_add(t, ff_shfl_xor(t, 4));
        t = ff_add(t, ff_shfl_xor(t, 2));
        t = ff_add(t, ff_shfl_xor(t, 1));
#pragma unroll
        for (int c = 0; c < 4; ++c)
            s[c] = FF{__shfl_sync(0xffffffffu, t.hi, 8 * c), __shfl_sync(0xffffffffu, t.lo, 8 * c)};
    };

    // ---------------- what eoc_prepare_kernel left: r_0 = p_0 = rhs_e, the diagonals
    const float4* const rhs = reinterpret_cast<const float4*>(S.x + 4 * (size_t)S.V);   // after chi_e
    float4 x[U], r[U], p[U], v[U], w[U];   // w: then u, then q
    E lo = {}, hi = {};
    constexpr std::true_type kDag = {};
    constexpr std::false_type kNoDag = {};
#pragma unroll
    for (int u = 0; u < U; ++u) {
        x[u] = v[u] = w[u] = r[u] = f4_zero();
        if (u < on) r[u] = rhs[2 * (size_t)((r0 + o0 + u) * Nh + i)];
        p[u] = r[u];
    }
    for (int h = tid; h < 4 * Nh; h += kN) {
        const int m = r0 * Nh + (h < 2 * Nh ? h - 2 * Nh : h - 2 * Nh + rows * Nh);
        const bool across = m < 0 || m >= S.V;
        const float4 q = rhs[2 * (size_t)(m < 0 ? m + S.V : m >= S.V ? m - S.V : m)];
        RH[h] = PH[h] = f4_mul(across ? -1.f : 1.f, q);
    }
    for (int h = tid; h < (rows + 2) * Nh; h += kN) {
        const int m = (r0 - 1) * Nh + h;
        const FF d = ld_ff1(S.dinv, m < 0 ? m + S.V : m >= S.V ? m - S.V : m);
        dih[h] = d.hi;
        dil[h] = d.lo;
        if (h < rows * Nh) {
            const FF e = ld_ff1(reinterpret_cast<const double*>(S.v32), r0 * Nh + h);
            deh[h] = e.hi;
            del[h] = e.lo;
        }
    }
    cluster_barrier();   // every CTA of the cluster has started: its shared memory can be written
    diagonals();
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (u < on) publish(kNoDag, u, p[u]);
    if (warp == 0) {
        FF t = {0.f, 0.f};   // |eta|^2: the tiles' sums in the same order in every CTA
        for (int q = lane; q < S.ntiles; q += 32) {
            const float2 f = a.partial[S.tile0 + q].f[0];
            t = ff_add(t, FF{f.x, f.y});
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t = ff_add(t, ff_shfl_xor(t, o));
        if (lane == 0) {
            st = EcState{};
            st.rr_ref = dbl_of(t);   // the rule of the full solve: relative to |eta|^2
            st.stop2 = a.stop2 ? a.stop2[S.rhs] : a.tol * a.tol * (a.tol_mode == YK_TOL_ABS ? 1.0 : st.rr_ref);
            st.stop2f = fmaxf((float)st.stop2, FLT_MIN);
            st.delta2 = (float)(a.reliable_delta * a.reliable_delta);
            st.due = a.reliable_every;
            st.rr_min = FLT_MAX;
            st.stray = -1;
        }
    }
    __syncthreads();

    // an update, from the thread's registers and back into them
    auto update = [&](float al, bool only_odd) {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < on) {
                V[je + u * Nh] = v[u];
                W[je + u * Nh] = x[u];
                g.p_own[(r0 + o0 + u) * Nh + i] = p[u];
            }
        for (int h = tid; h < 4 * Nh; h += kN) QH[h] = PH[h];
        const float4 s = ec_update<R1>(g, al, only_odd, rff);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            x[u] = r[u] = p[u] = f4_zero();
            if (u < on) {
                r[u] = V[je + u * Nh];
                p[u] = g.p_own[(r0 + o0 + u) * Nh + i];
            }
        }
        return s;
    };

    // (How far apart CTAs can be: one reaches its sends of iteration k + 1 only with
    // every CTA's sums of iteration k and, to QH, its neighbours' v of k + 1, so what
    // it overwrites has been read; the sums alternate between two places.)
    for (int k = 0;; ++k) {
        if (tid == 0) {
            mb_expect(mb0, 64u * (unsigned)Nh);
            mb_expect(mb0 + 8, 64u * (unsigned)Nh);
            mb_expect(mb0 + 16 + 8 * (k & 1), 32u * nc);
        }
        // ---------------- w, v
        odd_pass(kNoDag, p, PH, w, lo, hi);
        __syncthreads();
        even_pass(kNoDag, p, w, lo, hi, [&](int u, float4 h) {
            v[u] = h;
            publish(kDag, u, h);
            send_halo(VH, 0, u, edge_p(u), edge_n(u), h);
        });
        __syncthreads();
        // ---------------- u, q
        if (fs || ls) mb_wait(mb0, k & 1, &s_dead);
        odd_pass(kDag, v, VH, w, lo, hi);
        __syncthreads();
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
        even_pass(kDag, v, w, lo, hi, [&](int u, float4 h) {
            w[u] = h;
            send_halo(QH, 1, u, edge_p(u), edge_n(u), h);
            s4[0] = f4_dot(r[u], r[u], s4[0]);
            s4[1] = f4_dot(h, h, s4[1]);
            s4[2] = f4_dot(v[u], v[u], s4[2]);
            s4[3] = f4_dot(r[u], h, s4[3]);
        });
        partials(s4, k & 1, true);
        // ---------------- the scalar step (fast_step, yk_cg.cu), on the FP32 pipes
        if (warp == 0) {
            mb_wait(mb0 + 16 + 8 * (k & 1), (k >> 1) & 1, &s_dead);
            __syncwarp();
            FF t[4];
            totals(t, k & 1);
            if (lane == 0) {
                const float rr = t[0].hi + t[0].lo;
                float alpha = __fdividef(rr, t[2].hi + t[2].lo);
                int mode = kEcDone, status = 0, converged = 0;
                if (k == 0) st.rmax2 = rr;
                if (*(volatile int*)&s_dead) {
                    status = YK_ETIMEOUT;
                    *a.err = YK_ETIMEOUT;
                } else if (!isfinite(rr)) {
                    status = YK_ENAN;
                } else if (k == 0 && (st.stop2 < 0.0 || !(dbl_of(t[0]) > st.stop2))) {
                    if (st.stop2 < 0.0)
                        status = YK_ENOCONV;   // out of reach from the start
                    else
                        converged = 1;
                } else if (k >= a.max_iter) {
                    status = YK_ENOCONV;
                } else if (!isfinite(alpha) && rr > st.stop2f) {
                    status = YK_ENAN;
                } else {
                    const bool broken = !isfinite(alpha);   // p -> 0 below the stop: update without this step
                    if (broken) alpha = 0.f;
                    // |r - alpha q|^2: its terms cancel
                    const FF w = ff_mul(ff_add(FF{2.f * t[3].hi, 2.f * t[3].lo}, ff_neg(ff_mul(t[1], alpha))), alpha);
                    const FF ef = ff_add(t[0], ff_neg(w));
                    float est = ef.hi + ef.lo;
                    if (!(est > 0.f)) est = 0.f;
                    const float rmax2 = fmaxf(st.rmax2, rr), stop2f = st.stop2f;
                    st.rmax2 = rmax2;
                    st.rr_prev = rr;
                    const bool met = !(rr > stop2f) || !(est > stop2f);
                    bool ru = met || est < st.delta2 * rmax2 || broken || k + 1 >= a.max_iter;
                    if (a.reliable_every > 0) {
                        const int due = st.due - 1;
                        ru = ru || due == 0;
                        st.due = due == 0 ? a.reliable_every : due;
                    }
                    mode = ru ? kEcRu : kEcStep;
                    st.alpha = alpha;
                    st.beta = __fdividef(est, rr);
                    if (ru) st.est = met ? 0.f : est;
                }
                st.mode = mode;
                st.ru = 0;
                st.iters = k;
                if (mode == kEcDone) {
                    st.rr = dbl_of(t[0]);
                    st.status = status;
                    st.converged = converged;
                }
            }
        }
        __syncthreads();
        int mode = st.mode;
        // the neighbours' q: before its halo is read, or used for something else
        if (tid < 4 * Nh || mode != kEcStep) mb_wait(mb0 + 8, k & 1, &s_dead);
        if (mode == kEcDone) break;
        if (mode == kEcRu) {
            // ---------------- reliable update of chi_{e, k+1} in float-float
            const float4 s2 = update(st.alpha, false);
            const FF f4[4] = {{s2.x, s2.y}, {0.f, 0.f}, {s2.z, s2.w}, {0.f, 0.f}};
            partials(f4, k & 1, false);
            cluster_barrier();
            if (warp == 0) {
                FF t[4];
                totals(t, k & 1);
                if (lane == 0) {
                    const double rd = dbl_of(t[0]);
                    const float rf = (float)rd, rp = st.rr_prev;
                    st.mode = kEcDone;
                    st.ru = 1;
                    st.rr = rd;
                    st.iters = k + 1;
                    ++st.n_ru;
                    if (!isfinite(rd)) {
                        st.status = YK_ENAN;
                    } else if (!(rd > st.stop2)) {
                        st.converged = 1;
                    } else if (k + 1 >= a.max_iter) {
                        st.status = YK_ENOCONV;
                    } else if (a.stop2 && falls_no_further(st, k, rf)) {
                        st.status = YK_ENOCONV;
                    } else {
                        // p = r + beta (p - gamma r), gamma = <r, p> / |r|^2 (scalar_step);
                        // the divisions in FP32 where its range allows
                        if (rf > FLT_MIN && rp > FLT_MIN && rf < FLT_MAX && rp < FLT_MAX) {
                            const float b = rf / rp;
                            st.beta = b;
                            st.c_re = 1.f - b * ((t[2].hi + t[2].lo) * (1.f / rf));
                        } else {
                            const double b = rd / (double)rp;
                            st.beta = (float)b;
                            st.c_re = (float)(1.0 - b * (dbl_of(t[2]) / rd));
                        }
                        st.mode = kEcRedo;
                        st.rmax2 = rf;
                    }
                }
            }
            __syncthreads();
            mode = st.mode;
            if (mode == kEcDone) break;
        }
        // ---------------- the next iteration's r and p
        const float beta = st.beta;
        if (mode == kEcStep) {
            const float al = st.alpha;
            if (on > 0) {
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (has(u)) {
                        x[u] = f4_fma(al, v[u], x[u]);
                        r[u] = f4_fma(-al, w[u], r[u]);
                        p[u] = f4_fma(beta, p[u], r[u]);
                        publish(kNoDag, u, p[u]);
                    }
            }
            for (int h = tid; h < 4 * Nh; h += kN) {
                const float4 rv = f4_fma(-al, QH[h], RH[h]);
                RH[h] = rv;
                PH[h] = f4_fma(beta, PH[h], rv);
            }
        } else {
            const float c = st.c_re;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (u < on) {
                    p[u] = f4_fma(beta, p[u], f4_mul(c, r[u]));
                    publish(kNoDag, u, p[u]);
                }
            for (int h = tid; h < 4 * Nh; h += kN) PH[h] = f4_fma(beta, QH[h], f4_mul(c, RH[h]));
            diagonals();
        }
        __syncthreads();
    }
    // ---------------- chi for the force: chi_e is in x; the odd hop -A_o^-1
    // H^dag_oe chi_e, to which the force adds A_o^-1 eta_o, to t64 (both compact)
    if (!st.ru) {   // ended without an update: its odd hop is still to be formed
        update(0.f, true);
    }
    __syncthreads();
    for (int u = 0; u < on; ++u)
        st_ff(S.t64, (r0 + o0 + u) * Nh + i, ff_join(P[je + u * Nh], L[je + u * Nh]));
    if (rank == 0 && tid == 0) {
        CGState& o = *out_state;
        o.rr = st.rr;
        o.rr0 = st.rr_ref;
        o.rr_prev = (double)st.rr_prev;
        o.stop2 = st.stop2;
        o.rmax2 = (double)st.rmax2;
        o.active = 0;
        o.iters = st.iters;
        o.converged = st.converged;
        o.status = st.status;
        o.n_ru = st.n_ru;
        o.mode = 0;
        o.chi_ready = 2;   // however the solve ended
    }
    if (cluster_end(nc, &s_dead, &s_left, a.err) && rank == 0 && tid == 0) {
        CGState& o = *out_state;
        o.converged = 0;
        o.status = YK_ETIMEOUT;
    }
}

// ---------------------------------------------------------------------------
// A x = b for a complex b by two solves with D^dag of its real and imaginary
// planes (D is real): A = D^dag D, x = D^-1 (D^dag)^-1 b, and A = D D^dag with the
// factors exchanged.  A solve with D is one with D^dag too: with e = i gamma5 =
// [[0, 1], [-1, 0]] on spin, e D e^-1 = D^dag (gamma5 = sigma_2 changes the sign of
// both gammas), so D x = c is D^dag (e x) = e c.  An iteration of the Schur
// system costs half of one of A and there are 2.3 times fewer in each solve.
//
// Targets: |b - A x| <= |rho_1| + |D| |rho_2| with the residuals of the two solves,
// so the first goes to half the caller's target, the second to half of it over
// a bound of |D| (the largest diagonal, and 1 + r for each direction's hops).  The
// source is scaled by a power of two to norm 1 .. 2: the sums are FP32's.  The caller
// checks the residual of the result in FP64.
//
// The solves' residuals are float-float's, which fall no further than about 2^-46 of |b|
// (young fields of 192 x 128: 8e-15 at m0 = 0.1, 1.5e-14 at 0.02).  A second target below that is not
// tried (a negative target: the solve ends before its first iteration), nor the second solve
// after a first that failed, and a solve ends when its residual falls no further.  Without these
// the planes ran to the iteration cap before the other solve began: 192 x 128, tol 1e-13, a
// cap of 2000, 9.2 ms, where the other solve alone takes 3.4 (so 3.5).
// ---------------------------------------------------------------------------
namespace {

constexpr int kPlaneBlocks = 64;
constexpr double kPlaneReach = 0x1p-46;

__device__ __forceinline__ void eps_apply(double (&v)[4], int how)   // 1: e, -1: e^-1
{
    if (how == 0) return;
    for (int f = 0; f < 4; f += 2) {
        const double u = v[f], d = v[f + 1];
        v[f] = how > 0 ? d : -d;
        v[f + 1] = how > 0 ? -u : u;
    }
}

}  // namespace

// kPlaneBlocks partials of |b - t|^2 (t null: of |b|^2), then of the largest diagonal
__global__ void __launch_bounds__(kBlock) plane_norm_kernel(const double* __restrict__ b, const double* __restrict__ t,
                                                            const double* __restrict__ sigma, int V, double diag0,
                                                            double g, double* __restrict__ out)
{
    __shared__ double red[64];
    double s = 0.0, m = 0.0;
    for (int n = blockIdx.x * kBlock + threadIdx.x; n < V; n += kPlaneBlocks * kBlock) {
        const Site<double, 2> v = load_site<double, 2>(b, n);
        if (t) {
            const Site<double, 2> w = load_site<double, 2>(t, n);
#pragma unroll
            for (int q = 0; q < 8; ++q) s = fma(v.v[q] - w.v[q], v.v[q] - w.v[q], s);
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) s = fma(v.v[q], v.v[q], s);
            m = fmax(m, fabs(fma(g, sigma[n], diag0)));
        }
    }
    s = block_sum(s, red);
    m = block_max(m, red);
    if (threadIdx.x == 0) {
        out[blockIdx.x] = s;
        out[kPlaneBlocks + blockIdx.x] = m;
    }
}

// The planes of b, scaled, into the sources of the two real systems; the targets
// of the two solves (stop2[0 .. 1] and [2 .. 3]) and the scale (stop2[4]).
__global__ void __launch_bounds__(kBlock) plane_split_kernel(const double* __restrict__ b, const SysDev* __restrict__ sys,
                                                             const double* __restrict__ norm, double tol, int abs_tol,
                                                             int how, double hops, double* __restrict__ stop2)
{
    __shared__ double s_scale;
    if (threadIdx.x < 32) {
        double s = norm[threadIdx.x] + norm[threadIdx.x + 32];
        double m = fmax(norm[kPlaneBlocks + threadIdx.x], norm[kPlaneBlocks + 32 + threadIdx.x]);
        s = warp_sum(s);
        m = warp_max(m);
        if (threadIdx.x == 0) {
            double f = 1.0;
            if (s > 0.0 && isfinite(s)) f = scalbn(1.0, -(ilogb(s) >> 1));
            s_scale = f;
            if (blockIdx.x == 0) {
                const double b2 = s * f * f, t2 = abs_tol ? tol * f * (tol * f) : tol * tol * b2, d = m + hops;
                double t = t2 / 8.0, td = t2 / (8.0 * d * d);   // (half the target)^2, shared by the planes
                if (td < kPlaneReach * kPlaneReach * b2) t = td = -1.0;
                stop2[0] = stop2[1] = t;
                stop2[2] = stop2[3] = td;
                stop2[4] = f;
            }
        }
    }
    __syncthreads();
    const int n = blockIdx.x * kBlock + threadIdx.x;
    if (n >= sys[0].V) return;
    const double f = s_scale;
    const Site<double, 2> v = load_site<double, 2>(b, n);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        double q[4] = {f * v.v[k], f * v.v[2 + k], f * v.v[4 + k], f * v.v[6 + k]};
        eps_apply(q, how);
        store_site<double, 1>(sys[k].b, n, Site<double, 1>{{q[0], q[1], q[2], q[3]}});
    }
}

// The solution of a solve with D^dag at full site n of plane system S (E its compact
// view), as cg_eoc_kernel left it.
__device__ __forceinline__ void plane_solution(const SysDev& S, const SysDev& E, int n, double (&v)[4])
{
    const bool odd = (n / S.Nx + n) & 1;
    SiteFF c = ld_ff(odd ? S.t64 : S.x, n >> 1);
    if (odd) {
        const FF inv = ld_ff1(E.dinv, n >> 1);
        const Site<double, 1> b = load_site<double, 1>(S.b, n);
#pragma unroll
        for (int q = 0; q < 4; ++q) c.v[q] = ff_add(ff_mul(ff_split(b.v[q]), inv), c.v[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = dbl_of(c.v[q]);
}

// Between the solves: the first one's solution becomes the second one's source.
__global__ void __launch_bounds__(kBlock) plane_mid_kernel(const SysDev* __restrict__ sys, const SysDev* __restrict__ eo,
                                                           int how, const CGState* __restrict__ st, double* __restrict__ stop2)
{
    const int n = blockIdx.x * kBlock + threadIdx.x, k = blockIdx.y;
    if (n == 0 && !(st[0].converged && st[1].converged)) stop2[2 + k] = -1.0;
    if (n >= sys[k].V) return;
    double v[4];
    plane_solution(sys[k], eo[k], n, v);
    eps_apply(v, how);
    store_site<double, 1>(sys[k].b, n, Site<double, 1>{{v[0], v[1], v[2], v[3]}});
}

__global__ void __launch_bounds__(kBlock) plane_join_kernel(const SysDev* __restrict__ sys, const SysDev* __restrict__ eo,
                                                            int how, const double* __restrict__ stop2,
                                                            double* __restrict__ x)
{
    const int n = blockIdx.x * kBlock + threadIdx.x;
    if (n >= sys[0].V) return;
    const double f = 1.0 / stop2[4];   // a power of two
    Site<double, 2> o;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        double v[4];
        plane_solution(sys[k], eo[k], n, v);
        eps_apply(v, how);
#pragma unroll
        for (int q = 0; q < 4; ++q) o.v[2 * q + k] = f * v[q];
    }
    store_site<double, 2>(x, n, o);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {

const void* eoc_fn(const EocForm& f)
{
    if (!f.r1) return (const void*)cg_eoc_kernel<kEcMaxU, false, false>;
    switch (2 * f.u + (f.full ? 1 : 0)) {
        case 2: case 3: return (const void*)cg_eoc_kernel<1, true, true>;
        case 4: return (const void*)cg_eoc_kernel<2, false, true>;
        case 5: return (const void*)cg_eoc_kernel<2, true, true>;
        case 6: return (const void*)cg_eoc_kernel<3, false, true>;
        case 7: return (const void*)cg_eoc_kernel<3, true, true>;
        case 8: return (const void*)cg_eoc_kernel<4, false, true>;
        default: return (const void*)cg_eoc_kernel<4, true, true>;
    }
}

// Opts every form in to its cluster size and shared memory; the largest cluster
// that can be resident (16, or 8 where a GPC holds no 16; 0: none).
int eoc_max_cluster()
{
    return once_per_device([] {
        int best = kEcMaxC;
        for (int q = 0; q <= 2 * kEcMaxU; ++q) {
            const void* fn = eoc_fn({1, 1 + q / 2, 0, 0, q < 2 * kEcMaxU, q % 2 != 0});
            if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
                cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEocMaxSmem) != cudaSuccess) {
                cudaGetLastError();
                return 0;
            }
            for (int c = best;; c /= 2) {
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3(c);
                cfg.blockDim = dim3(kEcThreads);
                cfg.dynamicSmemBytes = kEocMaxSmem;
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
                    best = c;
                    break;
                }
                if (c <= 8) return 0;
            }
        }
        return best;
    });
}

// The form of a lattice on clusters of c CTAs.
bool form_at(int Nt, int Nh, double r, int c, EocForm* f)
{
    if (c > eoc_max_cluster() || Nt < 2 * c || Nh > kEcThreads / 2) return false;
    const int rows = (Nt + c - 1) / c, ns = kEcThreads / Nh;
    f->c = c;
    f->u = (rows + ns - 1) / ns;
    f->r1 = r == 1.0;
    // every thread with rows has u of them
    f->full = f->r1 && (f->u == 1 || (Nt % c == 0 && rows % f->u == 0));
    f->cells = (rows + 4) * Nh;
    f->nh = Nh;
    return f->u <= kEcMaxU && eoc_smem(*f) <= kEocMaxSmem;
}

}  // namespace

void cg_eoc_init() { eoc_max_cluster(); }

// Nt x Nh: the compact lattice.  The smallest cluster that holds a system, and up
// to `spread` times that while a CTA keeps 128 sites: with fewer the barriers and
// latencies of an iteration stay and nothing is saved (us a step, 32 x 32 on 1, 4
// and 8 CTAs: 96.4, 91.1, 90.5; 64 x 64 on 4, 8 and 16: 94.9, 90.9, 91.2).
bool cg_eoc_form(int Nt, int Nh, double r, int spread, EocForm* f)
{
    int c = 1;
    while (c <= kEcMaxC && !form_at(Nt, Nh, r, c, f)) c *= 2;
    if (c > kEcMaxC) return false;
    for (; spread > 1 && Nt * Nh >= 2 * c * 128; spread /= 2) {
        EocForm g;
        if (!form_at(Nt, Nh, r, 2 * c, &g)) break;
        c *= 2;
        *f = g;
    }
    return true;
}

static CGArgs eoc_args(const CGArgs& a)
{
    CGArgs b = a;
    b.sys_full = a.sys;
    b.sys = a.sys_eo;
    return b;
}

cudaError_t launch_eoc_prepare(const CGArgs& a, bool r1, bool other, int max_nh, cudaStream_t stream, bool first)
{
    const CGArgs b = eoc_args(a);
    const int n = a.tile_end - a.tile_begin;
    const size_t smem = 2 * sizeof(float4) * (kTile + 2 * (size_t)max_nh);
    int* const err = first ? b.err : nullptr;
    if (r1) eoc_prepare_kernel<true><<<n, kTile, smem, stream>>>(b, err);
    if (other) eoc_prepare_kernel<false><<<n, kTile, smem, stream>>>(b, err);
    return cudaGetLastError();
}

cudaError_t launch_cg_eoc(const CGArgs& a, const EocForm& f, const int* order, int count, cudaStream_t stream)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(f.c * count);
    cfg.blockDim = dim3(kEcThreads);
    cfg.dynamicSmemBytes = eoc_smem(f);
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = f.c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CGArgs b = eoc_args(a);
    int cells = f.cells, first = eoc_first_cells(f);
    void* args[] = {&b, &order, &cells, &first};
    return cudaLaunchKernelExC(&cfg, eoc_fn(f), args);
}

size_t plane_norm_doubles() { return 2 * kPlaneBlocks; }

// Whether a relative target is below what launch_plane_solve tries, whatever the field: |D| is
// bounded by more than the hops' part.
bool plane_out_of_reach(double tol, double r) { return tol < kPlaneReach * sqrt(8.0) * 2.0 * (1.0 + fabs(r)); }

// a: the two plane systems (a.sys, a.sys_eo, their tiles, a.st four states); norm,
// stop2: device scratch of plane_norm_doubles() and 5; tmp: two complex vectors.
// Leaves x, and in norm the partials of |b|^2, in resid those of |b - A x|^2.
cudaError_t launch_plane_solve(const CGArgs& a0, const EocForm& f, const double* b, double* x, const double* sigma, int Nt,
                               int Nx, double m0, double g, double r, double* norm, double* resid, double* stop2,
                               double* tmp, cudaStream_t stream)
{
    const int V = Nt * Nx, blocks = (V + kBlock - 1) / kBlock;
    const bool normal = a0.mtype == YK_NORMAL;
    CGArgs a = a0;
    a.mtype = YK_DAGGER;
    plane_norm_kernel<<<kPlaneBlocks, kBlock, 0, stream>>>(b, nullptr, sigma, V, 2.0 * r + m0, g, norm);
    plane_split_kernel<<<blocks, kBlock, 0, stream>>>(b, a.sys, norm, a.tol, a.tol_mode == YK_TOL_ABS, normal ? 1 : 0,
                                                      2.0 * (1.0 + fabs(r)), stop2);
    for (int stage = 0; stage < 2; ++stage) {
        a.st = a0.st + 2 * stage;
        a.stop2 = stop2 + 2 * stage;
        cudaError_t e = launch_eoc_prepare(a, f.r1, !f.r1, f.nh, stream, stage == 0);
        if (e == cudaSuccess) e = launch_cg_eoc(a, f, nullptr, 2, stream);
        if (e != cudaSuccess) return e;
        if (stage == 0) plane_mid_kernel<<<dim3(blocks, 2), kBlock, 0, stream>>>(a.sys, a.sys_eo, normal ? -1 : 1, a0.st, stop2);
    }
    plane_join_kernel<<<blocks, kBlock, 0, stream>>>(a.sys, a.sys_eo, normal ? 0 : -1, stop2, x);
    double* const t1 = tmp + 8 * (size_t)V;
    cudaError_t e = launch_dirac(x, tmp, sigma, Nt, Nx, m0, g, r, normal ? 1 : 0, YK_FP64, 2, stream, nullptr);
    if (e == cudaSuccess) e = launch_dirac(tmp, t1, sigma, Nt, Nx, m0, g, r, normal ? 0 : 1, YK_FP64, 2, stream, nullptr);
    if (e != cudaSuccess) return e;
    plane_norm_kernel<<<kPlaneBlocks, kBlock, 0, stream>>>(b, t1, sigma, V, 0.0, 0.0, resid);
    return cudaGetLastError();
}

}  // namespace yk

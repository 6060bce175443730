// yk_dirac.cu -- stand-alone Wilson-Dirac apply (the replacement for
// DiracOP<double>::applyD, code/src/Dirac.cu:23-70 and :144-190).
//
// One pass: a thread takes a site and walks its column in t through a band of
// rows, with rows t - 1, t, t + 1 in registers and row t + 2 on its way, so that
// every site is read from memory about once; the x neighbours come from the next
// lanes by warp shuffles (the lanes at a warp's and a row's ends load theirs).  The
// columns of all bands are dealt out to the threads one after another, so that narrow lattices
// leave no lanes idle (4096 x 2, FP64: 73.8 us with blocks of their own for each band, 7.6 so).  The
// antiperiodic time signs and neighbour indices are computed instead of read from
// IUP/IDN tables, and the output is written once (the reference zeroes `out`, adds
// the diagonal and adds the hops in three grid-synced passes).  Complex (K = 2)
// applies add the pion term g i gamma5 tau.pi when the chain carries pions.
//
// FP32 is bound by HBM (2048 x 2048: 45.1 us, 6.7 TB/s; its diagonal in float-float
// on the FP32 pipes), FP64 by its pipe, 1/64 of the FP32 rate: at r = 1 a time hop
// keeps one spin entry and an x hop a combination u -+ d, so that a spin pair and
// plane takes 8 operations against 14 (1000 x 749: 47.2 us against 87, of which
// the pipe needs 41).
#include "yk_cluster.cuh"
#include "yk_kernels.h"

namespace yk {

namespace {

template <typename R, int K>
__device__ __forceinline__ Unit<R, K> ld_unit(const R* base, int64_t i)
{
    Unit<R, K> s;
    const R* p = base + i * (2 * K);
    if constexpr (sizeof(R) * 2 * K == 8) {
        const float2 a = *reinterpret_cast<const float2*>(p);
        s.v[0] = a.x;
        s.v[1] = a.y;
    } else {
        constexpr int per = 16 / (int)sizeof(R);
#pragma unroll
        for (int q = 0; q < 2 * K / per; ++q) {
            const float4 a = reinterpret_cast<const float4*>(p)[q];
#pragma unroll
            for (int j = 0; j < per; ++j) s.v[q * per + j] = reinterpret_cast<const R*>(&a)[j];
        }
    }
    return s;
}

template <typename R, int K>
__device__ __forceinline__ void st_unit(R* base, int64_t i, const Unit<R, K>& s)
{
    R* p = base + i * (2 * K);
    if constexpr (sizeof(R) * 2 * K == 8) {
        *reinterpret_cast<float2*>(p) = make_float2((float)s.v[0], (float)s.v[1]);
    } else {
        constexpr int per = 16 / (int)sizeof(R);
#pragma unroll
        for (int q = 0; q < 2 * K / per; ++q) {
            float4 a;
#pragma unroll
            for (int j = 0; j < per; ++j) reinterpret_cast<R*>(&a)[j] = s.v[q * per + j];
            reinterpret_cast<float4*>(p)[q] = a;
        }
    }
}

// What an x neighbour passes on: at r = 1 the spin combination its hop keeps
// (K numbers), else both spin entries.
template <typename R, int K, bool R1>
struct XPart {
    R v[R1 ? K : 2 * K];
};

template <typename R, int K, bool R1>
__device__ __forceinline__ XPart<R, K, R1> x_part(const Unit<R, K>& c, R s)   // u + s d
{
    XPart<R, K, R1> o;
#pragma unroll
    for (int k = 0; k < (R1 ? K : 2 * K); ++k) o.v[k] = R1 ? fma(s, c.v[K + k], c.v[k]) : c.v[k];
    return o;
}

// -c where `yes`.  In FP64 by the sign bits: lanes differ, and a negation that is selected
// takes the FP64 pipe in all of them (1000 x 749: 58.6 us against 47.3; FP32 has it for nothing).
template <typename R, int K>
__device__ __forceinline__ void negate_if(Unit<R, K>& c, bool yes)
{
    const unsigned m = yes ? 0x80000000u : 0u;
#pragma unroll
    for (int k = 0; k < 2 * K; ++k) {
        if constexpr (sizeof(R) == 8)
            c.v[k] = __hiloint2double((int)((unsigned)__double2hiint(c.v[k]) ^ m), __double2loint(c.v[k]));
        else
            c.v[k] = yes ? -c.v[k] : c.v[k];
    }
}

}  // namespace

template <typename R, int K, bool DAG, bool R1>
__global__ void __launch_bounds__(kBlock) dirac_kernel(const R* __restrict__ in, R* __restrict__ out,
                                                       const double* __restrict__ sigma, const double* __restrict__ pi,
                                                       int Nt, int Nx, int columns, int band, double diag0, double g,
                                                       double r, float4 ff)
{
    using Un = Unit<R, K>;
    constexpr int F = 2;   // flavours
    const int V = Nt * Nx, lane = threadIdx.x & 31;
    const int at = blockIdx.x * kBlock + threadIdx.x;
    if (at - lane >= columns) return;
    const int col = min(at, columns - 1);   // the last warp's lanes past the last column repeat its work
    const int by = col / Nx, x = col - by * Nx;
    // the x neighbours come from the lanes but at the ends
    const bool ld_up = lane == 31 || x == Nx - 1, ld_dn = lane == 0 || x == 0;
    const int x_up = x == Nx - 1 ? 0 : x + 1, x_dn = x == 0 ? Nx - 1 : x - 1;
    const int t0 = by * band, t1 = min(t0 + band, Nt);
    const R rr = (R)r, half = R(0.5), s = DAG ? R(-1) : R(1);
    const FF gf = {ff.x, ff.y}, df = {ff.z, ff.w};
    struct Part {
        Un u[F];
    };
    auto load = [&](int t, int j) {
        Part p;
        const int64_t o = ((int64_t)(t < 0 ? t + Nt : t >= Nt ? t - Nt : t) * Nx + j) * F;
#pragma unroll
        for (int q = 0; q < F; ++q) p.u[q] = ld_unit<R, K>(in, o + q);
        return p;
    };
    Part prev = load(t0 - 1, x), cur = load(t0, x), next = load(t0 + 1, x);
    double sg = sigma[t0 * Nx + x];
#pragma unroll
    for (int q = 0; q < F; ++q) negate_if(prev.u[q], t0 == 0);
    // as many rows in every lane, for the shuffles: those past a shorter last band are not stored
    for (int k = 0; k < band; ++k) {
        const int t = t0 + k, n = min(t, Nt - 1) * Nx + x;
        Part ahead = next;
        double sg_ahead = sg;
        if (t + 1 < t1) {
            ahead = load(t + 2, x);
            sg_ahead = sigma[n + Nx];
        }
        XPart<R, K, R1> up[F], dn[F];
#pragma unroll
        for (int q = 0; q < F; ++q) negate_if(next.u[q], t + 1 == Nt);
        if constexpr (sizeof(R) == 4) {
#pragma unroll
            for (int q = 0; q < F; ++q) {
                up[q] = x_part<R, K, R1>(cur.u[q], -s);
                dn[q] = x_part<R, K, R1>(cur.u[q], s);
#pragma unroll
                for (int k = 0; k < (R1 ? K : 2 * K); ++k) {
                    up[q].v[k] = __shfl_down_sync(0xffffffffu, up[q].v[k], 1);
                    dn[q].v[k] = __shfl_up_sync(0xffffffffu, dn[q].v[k], 1);
                }
            }
            if (ld_up) {
                const Part e = load(t, x_up);
#pragma unroll
                for (int q = 0; q < F; ++q) up[q] = x_part<R, K, R1>(e.u[q], -s);
            }
            if (ld_dn) {
                const Part e = load(t, x_dn);
#pragma unroll
                for (int q = 0; q < F; ++q) dn[q] = x_part<R, K, R1>(e.u[q], s);
            }
        } else {
            // the neighbours' sites first, so that the ends' combinations cost no FP64
            // instructions of their own
            auto shifted = [&](bool down) {
                Part e;
#pragma unroll
                for (int q = 0; q < F; ++q)
#pragma unroll
                    for (int k = 0; k < 2 * K; ++k)
                        e.u[q].v[k] = down ? __shfl_down_sync(0xffffffffu, cur.u[q].v[k], 1)
                                           : __shfl_up_sync(0xffffffffu, cur.u[q].v[k], 1);
                if (down ? ld_up : ld_dn) e = load(t, down ? x_up : x_dn);
                return e;
            };
            const Part eu = shifted(true);
#pragma unroll
            for (int q = 0; q < F; ++q) up[q] = x_part<R, K, R1>(eu.u[q], -s);
            const Part ed = shifted(false);
#pragma unroll
            for (int q = 0; q < F; ++q) dn[q] = x_part<R, K, R1>(ed.u[q], s);
        }
        R diag;
        if constexpr (sizeof(R) == 4) {
            const FF sf = ff_split(sg), q = ff_add(df, ff_mul(gf, sf));
            diag = q.hi;
            // a field value or a coupling beyond FP32's range, in FP64 (asm: the compiler would
            // do so always and select)
            if (!isfinite(q.hi) || (sf.hi == 0.f && __double2hiint(sg) << 1 != 0))
                asm volatile("{\n\t.reg .f64 d;\n\tfma.rn.f64 d, %1, %2, %3;\n\tcvt.rn.f32.f64 %0, d;\n\t}"
                             : "=f"(diag)
                             : "d"(g), "d"(sg), "d"(diag0));
        } else {
            diag = fma(g, sg, diag0);
        }
        Part o;
#pragma unroll
        for (int q = 0; q < F; ++q) {
            const Un &c = cur.u[q], &tu = next.u[q], &td = prev.u[q];
            const XPart<R, K, R1>&xu = up[q], &xd = dn[q];
            if constexpr (R1) {
                // r = 1 (unit_dirac, yk_cg_small.cu): D keeps d of t + 1, u of t - 1, D^dag the others
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const R hu = DAG ? tu.v[k] : td.v[k], hd = DAG ? td.v[K + k] : tu.v[K + k];
                    o.u[q].v[k] = fma(-half, xu.v[k] + xd.v[k], fma(diag, c.v[k], -hu));
                    o.u[q].v[K + k] = fma(half * s, xu.v[k] - xd.v[k], fma(diag, c.v[K + k], -hd));
                }
            } else {
                // dirac_combine (yk_common.cuh)
                const R cp = -half * (rr + R(1)), cm = -half * (rr - R(1)), a = -half * rr, bx = half * s;
                const R uu = DAG ? cp : cm, ud = DAG ? cm : cp;   // of t + 1; t - 1 takes them exchanged
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const int u = k, d = K + k;
                    const R ou = fma(ud, td.v[u], fma(uu, tu.v[u], diag * c.v[u]));
                    const R od = fma(uu, td.v[d], fma(ud, tu.v[d], diag * c.v[d]));
                    o.u[q].v[u] = fma(a, xu.v[u] + xd.v[u], fma(bx, xu.v[d] - xd.v[d], ou));
                    o.u[q].v[d] = fma(a, xu.v[d] + xd.v[d], fma(bx, xu.v[u] - xd.v[u], od));
                }
            }
        }
        if constexpr (K == 2)
            if (pi) {
                const double gs = DAG ? -g : g;
                const R s1 = (R)(gs * pi[n]), s2 = (R)(gs * pi[V + n]), s3 = (R)(gs * pi[2 * V + n]);
#pragma unroll
                for (int q = 0; q < F; ++q)
                    unit_pions<R>(o.u[q], cur.u[q], cur.u[F - 1 - q], q, s1, s2, s3);
            }
        if (at < columns && t < t1)
#pragma unroll
            for (int q = 0; q < F; ++q) st_unit<R, K>(out, (int64_t)n * F + q, o.u[q]);
        prev = cur;
        cur = next;
        next = ahead;
        sg = sg_ahead;
    }
}

template <typename R, int K, bool DAG, bool R1>
static cudaError_t launch_t(const void* in, void* out, const double* sigma, const double* pi, int Nt, int Nx,
                            double m0, double g, double r, cudaStream_t stream)
{
    // bands of up to four rows (two rows more are read for each, most of them from
    // L2: FP32, 2048 x 2048, in an early form four rows 51.4 us, eight 53.3, two 54.5), fewer
    // where the lattice would give each SM less than four blocks
    const int n_sm = once_per_device([] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 1;
    });
    int band = (int)((int64_t)Nt * Nx / (4 * kBlock * n_sm));
    band = band < 1 ? 1 : band > 4 ? 4 : band;
    if (band > Nt) band = Nt;   // (a lane past the last row wraps its loads once)
    const int columns = (Nt + band - 1) / band * Nx;
    // g and the diagonal's constant as float-float, by the host (NaN for a g that FP32 holds
    // with fewer bits or not at all: the kernel takes FP64 then)
    const double diag0 = 2.0 * r + m0;
    const float gh = g == 0.0 || (fabs(g) > 0x1p-100 && fabs(g) < 0x1p100) ? (float)g : NAN, dh = (float)diag0;
    const float4 ff = make_float4(gh, (float)(g - gh), dh, (float)(diag0 - dh));
    dirac_kernel<R, K, DAG, R1><<<(columns + kBlock - 1) / kBlock, kBlock, 0, stream>>>(
        (const R*)in, (R*)out, sigma, pi, Nt, Nx, columns, band, diag0, g, r, ff);
    return cudaGetLastError();
}

template <typename R, int K>
static cudaError_t launch_k(const void* in, void* out, const double* sigma, const double* pi, int Nt, int Nx,
                            double m0, double g, double r, int dagger, cudaStream_t stream)
{
    if (r == 1.0)
        return dagger ? launch_t<R, K, true, true>(in, out, sigma, pi, Nt, Nx, m0, g, r, stream)
                      : launch_t<R, K, false, true>(in, out, sigma, pi, Nt, Nx, m0, g, r, stream);
    return dagger ? launch_t<R, K, true, false>(in, out, sigma, pi, Nt, Nx, m0, g, r, stream)
                  : launch_t<R, K, false, false>(in, out, sigma, pi, Nt, Nx, m0, g, r, stream);
}

cudaError_t launch_dirac(const void* in, void* out, const double* sigma, int Nt, int Nx, double m0,
                         double g, double r, int dagger, int prec, int K, cudaStream_t stream, const double* pi)
{
    if (K == 1) pi = nullptr;   // pions need complex sites
    if (prec == YK_FP64)
        return K == 1 ? launch_k<double, 1>(in, out, sigma, pi, Nt, Nx, m0, g, r, dagger, stream)
                      : launch_k<double, 2>(in, out, sigma, pi, Nt, Nx, m0, g, r, dagger, stream);
    return K == 1 ? launch_k<float, 1>(in, out, sigma, pi, Nt, Nx, m0, g, r, dagger, stream)
                  : launch_k<float, 2>(in, out, sigma, pi, Nt, Nx, m0, g, r, dagger, stream);
}

}  // namespace yk

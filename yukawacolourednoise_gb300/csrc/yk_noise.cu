// yk_noise.cu -- coloured noise xi = Z2D(mask * D2Z(w)) / V of
// code/src/colouredNoise.cpp:155-178, rebuilt as three shared-memory FFT
// passes instead of RNG kernel + cuFFT D2Z + mask kernel + cuFFT Z2D:
//   1. rows:    Philox Gaussian white noise generated in registers, written
//               to shared memory, forward FFT along x, spectrum rows stored;
//               two real rows go through one complex FFT (w_t + i w_{t+1})
//               and are separated by the symmetry of real transforms;
//   2. columns: a strip of columns loaded once, forward FFT along t, sharp
//               momentum cutoff (and the 1/V normalisation of the reference's
//               mask), inverse FFT along t, stored back -- only strips that
//               hold a kept mode: a column kx keeps some mode exactly when it
//               keeps (0, kx), and the other columns come out zero;
//   3. rows:    inverse FFT along x of two rows at once (Y_t + i Y_{t+1}:
//               both results are real), written as xi.
// The real field is transformed as a complex one; since the cutoff is even
// in k, this equals the reference's r2c/c2r pair.
// When the cutoff keeps every mode (cutFraction >= 1) the filter is the
// identity and a single generation pass writes xi = w.
// Every chain of a context is handled by the same launches through
// block -> (chain, row / column strip) tables.
#include "yk_common.cuh"
#include "yk_kernels.h"

namespace yk {

__device__ __forceinline__ double2 c_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 c_sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 c_mul(double2 a, double2 w)
{
    return make_double2(fma(a.x, w.x, -a.y * w.y), fma(a.x, w.y, a.y * w.x));
}

// A stage of the transform below: sub-sequences of r n points out of n ones
// (m = n / r), s of them interleaved.  Butterfly b of a sequence takes elements
// b + j M (M = N / r); with b = p s + q its outputs, times w_n^{p k}, go to q + s (r p + k).
struct FftStage {
    const double2* x;
    double2* y;
    int N, M, lm, s, ls, sj, sc, nseq;   // M = 2^lm (lm < 0: no power of two)
    bool twiddle, inverse;
    const double2* tw;

    __device__ __forceinline__ double2 in(int b, int j, int c) const { return x[(b + j * M) * sj + c * sc]; }
    __device__ __forceinline__ double2 root(int k) const   // exp(-+2 pi i k / N), k < N
    {
        double2 w = tw[k];
        if (inverse) w.y = -w.y;
        return w;
    }
    // output k of a butterfly, as it is stored
    __device__ __forceinline__ void put(int p, int q, int r, int k, int c, double2 v) const
    {
        y[(q + s * (r * p + k)) * sj + c * sc] = v;
    }
    __device__ __forceinline__ void out(int p, int q, int r, int k, int c, double2 v) const
    {
        put(p, q, r, k, c, twiddle && k > 0 ? c_mul(v, root(p * k * s)) : v);
    }
};

// r = 4 or 2: the first stages, so that s is a power of two, 2^ls.  A butterfly's loads go
// before its arithmetic and its stores after it: a short transform is bound by their latency and
// that of integer divisions, and the compiler moves no twiddle's load over a store that may alias it
// (256 x 256, the noise in all: 43.0 us with each output's twiddle loaded at its store, 37.0 so).
__device__ __forceinline__ void fft_even(const FftStage& f, int r)
{
    for (int idx = threadIdx.x; idx < f.M * f.nseq; idx += blockDim.x) {
        const int c = f.lm >= 0 ? idx >> f.lm : idx / f.M, b = idx - c * f.M, p = b >> f.ls, q = b & (f.s - 1);
        double2 w[4];
        if (f.twiddle)
#pragma unroll
            for (int k = 1; k < 4; ++k)
                if (k < r) w[k] = f.root(p * k * f.s);
        const double2 a0 = f.in(b, 0, c), a1 = f.in(b, 1, c);
        if (r == 4) {
            const double2 a2 = f.in(b, 2, c), a3 = f.in(b, 3, c);
            const double2 t0 = c_add(a0, a2), t1 = c_sub(a0, a2), t2 = c_add(a1, a3), d = c_sub(a1, a3);
            const double2 t3 = f.inverse ? make_double2(-d.y, d.x) : make_double2(d.y, -d.x);
            double2 o[4] = {c_add(t0, t2), c_add(t1, t3), c_sub(t0, t2), c_sub(t1, t3)};
            if (f.twiddle)
#pragma unroll
                for (int k = 1; k < 4; ++k) o[k] = c_mul(o[k], w[k]);
#pragma unroll
            for (int k = 0; k < 4; ++k) f.put(p, q, 4, k, c, o[k]);
        } else {
            const double2 o = c_sub(a0, a1);
            f.put(p, q, 2, 0, c, c_add(a0, a1));
            f.put(p, q, 2, 1, c, f.twiddle ? c_mul(o, w[1]) : o);
        }
    }
}

// Outputs k and r - k of an odd r share their sums over a_j + a_{r-j} and a_j - a_{r-j}.
__device__ __forceinline__ void fft_odd(const FftStage& f, int r)
{
    const int h = r / 2, items = f.M * (h + 1);
    for (int idx = threadIdx.x; idx < items * f.nseq; idx += blockDim.x) {
        const int c = idx / items, e = idx - c * items, k = e / f.M, b = e - k * f.M, p = b / f.s, q = b - p * f.s;
        double2 R = f.in(b, 0, c), I = make_double2(0.0, 0.0);
        int t = 0;   // j k mod r
        for (int j = 1; j <= h; ++j) {
            t += k;
            if (t >= r) t -= r;
            const double2 u = f.in(b, j, c), v = f.in(b, r - j, c), w = f.root(t * f.M);
            const double2 S = c_add(u, v), D = c_sub(u, v);
            R.x = fma(w.x, S.x, R.x);
            R.y = fma(w.x, S.y, R.y);
            I.x = fma(-w.y, D.y, I.x);   // i sin D
            I.y = fma(w.y, D.x, I.y);
        }
        f.out(p, q, r, k, c, c_add(R, I));
        if (k > 0) f.out(p, q, r, r - k, c, c_sub(R, I));
    }
}

// FFT of `nseq` sequences of length N in shared memory; element j of sequence c
// is buf[j * sj + c * sc].  Radix 4, 2 and every odd prime of N, each stage from
// one of the two buffers into the other (self-sorting); returns the one that
// holds the result.  tw[k] = exp(-2 pi i k / N), k < N.  Bound by the FP64 pipe:
// a prime r costs about 4 r operations a point, so that a length with small
// factors is far from a direct sum's 4 N (the noise of a 160 x 224 step in all:
// 292 us by direct sums, 41 so).
__device__ double2* smem_fft(double2* buf, double2* tmp, int N, int nseq, int sj, int sc,
                             const double2* __restrict__ tw, bool inverse)
{
    int n = N, s = 1, ls = 0, prime = 3;
    while (n > 1) {
        int r;
        if (n % 4 == 0) {
            r = 4;
        } else if (n % 2 == 0) {
            r = 2;
        } else {
            while (n % prime) prime = prime * prime > n ? n : prime + 2;
            r = prime;
        }
        if (r & 1) {
            fft_odd(FftStage{buf, tmp, N, N / r, 0, s, 0, sj, sc, nseq, n > r, inverse, tw}, r);
            n /= r;
        } else {
            const int M = N >> (r >> 1), lm = (M & (M - 1)) == 0 ? __ffs(M) - 1 : -1;
            fft_even(FftStage{buf, tmp, N, M, lm, s, ls, sj, sc, nseq, n > r, inverse, tw}, r);
            n >>= r >> 1;
            ls += r >> 1;
        }
        __syncthreads();
        s *= r;
        double2* const q = buf;
        buf = tmp;
        tmp = q;
    }
    return buf;
}

__device__ __forceinline__ double white_at(const ChainDev& C, const double* given, int n)
{
    if (given) return given[n];
    const RngStream rs = rng_stream(C.seed, C.chain_id, (uint64_t)C.step, 1u, 0u);
    return normal_at(rs, (uint32_t)n);
}

// rows t and t + 1 (when t + 1 < Nt) of the white noise, transformed along x
// as one complex sequence w_t + i w_{t+1}; with Z its transform,
// W_t[k] = (Z[k] + conj Z[-k]) / 2 and W_{t+1}[k] = (Z[k] - conj Z[-k]) / 2i.
// Only the columns that keep a mode are stored.
__global__ void __launch_bounds__(kBlock) noise_rows_fwd(ChainDev* chains, const int2* rows, int nrows,
                                                         const double* given)
{
    extern __shared__ double2 sm[];
    for (int item = blockIdx.x; item < nrows; item += gridDim.x) {
    if (item != (int)blockIdx.x) __syncthreads();   // the previous item's reads of sm are done
    const int2 ct = rows[item];
    const ChainDev& C = chains[ct.x];
    const int Nx = C.Nx, t = ct.y;
    const bool two = t + 1 < C.Nt;
    double2* buf = sm;
    double2* tmp = sm + Nx;
    const int base = t * Nx;
    if (!given && (Nx & 3) == 0) {
        // four normals of each row per counter
        const RngStream rs = rng_stream(C.seed, C.chain_id, (uint64_t)C.step, 1u, 0u);
        for (int x4 = threadIdx.x; x4 < Nx / 4; x4 += blockDim.x) {
            const float4 z = normal4(rs, (uint32_t)((base >> 2) + x4));
            const float4 y = two ? normal4(rs, (uint32_t)(((base + Nx) >> 2) + x4)) : make_float4(0.f, 0.f, 0.f, 0.f);
            buf[4 * x4] = make_double2(z.x, y.x);
            buf[4 * x4 + 1] = make_double2(z.y, y.y);
            buf[4 * x4 + 2] = make_double2(z.z, y.z);
            buf[4 * x4 + 3] = make_double2(z.w, y.w);
        }
    } else {
        for (int x = threadIdx.x; x < Nx; x += blockDim.x)
            buf[x] = make_double2(white_at(C, given, base + x), two ? white_at(C, given, base + Nx + x) : 0.0);
    }
    __syncthreads();
    buf = smem_fft(buf, tmp, Nx, 1, 1, 0, C.tw_x, false);
    for (int k = threadIdx.x; k < Nx; k += blockDim.x) {
        if (!C.keep[k]) continue;   // the column keeps no mode
        const double2 zk = buf[k], zm = buf[k == 0 ? 0 : Nx - k];
        C.spec[base + k] = make_double2(0.5 * (zk.x + zm.x), 0.5 * (zk.y - zm.y));
        if (two) C.spec[base + Nx + k] = make_double2(0.5 * (zk.y + zm.y), 0.5 * (zm.x - zk.x));
    }
    }
}

__global__ void __launch_bounds__(kBlock) noise_cols(ChainDev* chains, const int2* cols, int ncols)
{
    extern __shared__ double2 sm[];
    for (int item = blockIdx.x; item < ncols; item += gridDim.x) {
    if (item != (int)blockIdx.x) __syncthreads();
    const int2 cc = cols[item];
    const ChainDev& C = chains[cc.x];
    const int Nt = C.Nt, Nx = C.Nx, x0 = cc.y;
    int cw = noise_strip(Nt);
    if (cw > Nx - x0) cw = Nx - x0;
    double2* buf = sm;
    double2* tmp = sm + Nt * cw;
    for (int idx = threadIdx.x; idx < Nt * cw; idx += blockDim.x) {
        const int t = idx / cw, c = idx - t * cw;
        buf[idx] = C.keep[x0 + c] ? C.spec[t * Nx + x0 + c] : make_double2(0.0, 0.0);   // unwritten otherwise
    }
    __syncthreads();
    if (double2* const q = smem_fft(buf, tmp, Nt, cw, cw, 1, C.tw_t, false); q != buf) {
        tmp = buf;
        buf = q;
    }
    const double inv = 1.0 / (double)C.V;
    for (int idx = threadIdx.x; idx < Nt * cw; idx += blockDim.x) {
        const int t = idx / cw, c = idx - t * cw;
        const double m = C.keep[t * Nx + x0 + c] ? inv : 0.0;
        buf[idx].x *= m;
        buf[idx].y *= m;
    }
    __syncthreads();
    buf = smem_fft(buf, tmp, Nt, cw, cw, 1, C.tw_t, true);
    for (int idx = threadIdx.x; idx < Nt * cw; idx += blockDim.x) {
        const int t = idx / cw, c = idx - t * cw;
        C.spec[t * Nx + x0 + c] = buf[idx];
    }
    }
}

// rows t and t + 1 of the filtered spectrum, inverse-transformed along x as
// one sequence Y_t + i Y_{t+1}: both results are real, so they come out as
// the real and imaginary parts.  Columns that keep no mode are zero.
__global__ void __launch_bounds__(kBlock) noise_rows_inv(ChainDev* chains, const int2* rows, int nrows)
{
    extern __shared__ double2 sm[];
    for (int item = blockIdx.x; item < nrows; item += gridDim.x) {
    if (item != (int)blockIdx.x) __syncthreads();
    const int2 ct = rows[item];
    const ChainDev& C = chains[ct.x];
    const int Nx = C.Nx, t = ct.y;
    const bool two = t + 1 < C.Nt;
    double2* buf = sm;
    double2* tmp = sm + Nx;
    for (int x = threadIdx.x; x < Nx; x += blockDim.x) {
        double2 v = make_double2(0.0, 0.0);
        if (C.keep[x]) {
            const double2 a = C.spec[t * Nx + x];
            const double2 b = two ? C.spec[(t + 1) * Nx + x] : make_double2(0.0, 0.0);
            v = make_double2(a.x - b.y, a.y + b.x);
        }
        buf[x] = v;
    }
    __syncthreads();
    buf = smem_fft(buf, tmp, Nx, 1, 1, 0, C.tw_x, true);
    for (int x = threadIdx.x; x < Nx; x += blockDim.x) {
        C.xi[t * Nx + x] = buf[x].x;
        if (two) C.xi[(t + 1) * Nx + x] = buf[x].y;
    }
    }
}

__global__ void __launch_bounds__(kBlock) noise_white(ChainDev* chains, const int2* tiles, const double* given)
{
    const int2 ct = tiles[blockIdx.x];
    const ChainDev& C = chains[ct.x];
    const int n = ct.y + threadIdx.x;
    if (n < C.V) C.xi[n] = white_at(C, given, n);
}

void noise_init_attributes()
{
    static bool attr_set = false;
    if (!attr_set) {
        const int big = (int)(2 * sizeof(double2) * kMaxFFT);
        cudaFuncSetAttribute(noise_rows_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
        cudaFuncSetAttribute(noise_cols, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
        cudaFuncSetAttribute(noise_rows_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
        attr_set = true;
    }
}

cudaError_t launch_noise_tables(ChainDev* d_chains, const NoiseTables& tb, int max_nx, int max_cols_elems,
                                const double* given, cudaStream_t stream, int max_blocks)
{
    noise_init_attributes();
    auto grid = [&](int n) { return (max_blocks > 0 && n > max_blocks) ? max_blocks : n; };
    if (tb.nwhite > 0) noise_white<<<tb.nwhite, kTile, 0, stream>>>(d_chains, tb.white, given);
    if (tb.nrows > 0) {
        const size_t rs = 2 * sizeof(double2) * (size_t)max_nx;
        const size_t cs = 2 * sizeof(double2) * (size_t)max_cols_elems;
        noise_rows_fwd<<<grid(tb.nrows), kBlock, rs, stream>>>(d_chains, tb.rows, tb.nrows, given);
        if (tb.ncols > 0) noise_cols<<<grid(tb.ncols), kBlock, cs, stream>>>(d_chains, tb.cols, tb.ncols);
        noise_rows_inv<<<grid(tb.nrows), kBlock, rs, stream>>>(d_chains, tb.rows, tb.nrows);
    }
    return cudaGetLastError();
}

}  // namespace yk

// DST-I through shared-memory FFTs, for grids with 2(n+1) a power of two (n = 31, 63, 127,
// 255, 511, 1023, 2047): the reference's fast Dirichlet solver evaluates the same transforms with
// real-to-complex repacking and cuFFT (FFTPoissonSolverDirichletFast.cpp:34-72, 196-328).
//
// Two real rows a, b (length n) are packed as one complex odd extension of length M = 2(n+1):
//   z[0] = z[n+1] = 0, z[j] = a[j-1] + i b[j-1], z[M-j] = -z[j]   (j = 1..n)
// whose DFT is Z[k] = -2i S(a)[k] + 2 S(b)[k] with S(v)[k] = sum_j v[j-1] sin(pi j k / (n+1)),
// i.e. the DST-I of both rows from one radix-2 FFT. A Poisson solve is three kernels:
//   x-pass (rows along x, transposed write)  ->  y-pass, eigenvalue divide, y-pass (transposed
//   write back)  ->  x-pass with the scatter into the field components.
#pragma once

#include <vector>

#include "common.cuh"

namespace hpq {

template <class R>
struct Cx {
    R re, im;
};

template <class R>
__device__ __forceinline__ Cx<R> cmul(const Cx<R>& v0, const Cx<R>& w) {
    return {v0.re * w.re - v0.im * w.im, v0.re * w.im + v0.im * w.re};
}

// ------------------------------------------------------------------------------------------
// The transform of a row pair: FFT of length M = 2(n+1) with 8 elements per thread in registers
// (Stockham autosort: radix-8 passes, then one of radix 8, 4 or 2), so that M = 2048 passes
// through shared memory 3 times; the in-place radix-2/4 form it replaces did 6 times and
// put its input in bit-reversed order first. Bound by shared memory (ncu at M = 2048: L1 and shared
// memory 80-84 %, FP64 pipe 16-18 %, DRAM 5-8 %); a 1023^2 solve of three fields takes 191 us in double
// and 134 us in single precision and took 469 and 323 us with that form.
// ------------------------------------------------------------------------------------------
// row pairs per block: blocks of at least 64 threads, four rows per block up to M = 2048 so that a
// transposed write covers 32 bytes in double
template <int M>
struct DstCfg {
    static constexpr int T = M / 8;                                   // threads per row pair
    static constexpr int F = M <= 256 ? 64 / T * 2 : M <= 2048 ? 2 : 1;  // row pairs per block
    static constexpr int RB = 2 * F;
    static constexpr int NT = F * T;
    static constexpr int MP = M + M / 8;                              // padded complex row
    template <class R>
    static constexpr size_t smem() { return (size_t)F * MP * sizeof(Cx<R>); }
};
// one word group of padding per 8 elements: the stride-8 writes of the first pass then touch
// different banks
__device__ __forceinline__ int dst_pad(int i) { return i + (i >> 3); }

// 8-point DFT (exp(-i)) in place, outputs in natural order
template <class R>
__device__ __forceinline__ void dft8(Cx<R> (&v)[8]) {
    const R h = R(0.70710678118654752440);
    auto bf = [](Cx<R>& a, Cx<R>& b) {
        const Cx<R> t = {a.re - b.re, a.im - b.im};
        a = {a.re + b.re, a.im + b.im};
        b = t;
    };
    bf(v[0], v[4]); bf(v[1], v[5]); bf(v[2], v[6]); bf(v[3], v[7]);
    // odd half times exp(-i pi q / 4)
    v[5] = {(v[5].re + v[5].im) * h, (v[5].im - v[5].re) * h};
    v[6] = {v[6].im, -v[6].re};
    v[7] = {(v[7].im - v[7].re) * h, -(v[7].re + v[7].im) * h};
    bf(v[0], v[2]); bf(v[1], v[3]); bf(v[4], v[6]); bf(v[5], v[7]);
    v[3] = {v[3].im, -v[3].re};
    v[7] = {v[7].im, -v[7].re};
    bf(v[0], v[1]); bf(v[2], v[3]); bf(v[4], v[5]); bf(v[6], v[7]);
    // v[bit-reversed] -> natural order
    Cx<R> t = v[1]; v[1] = v[4]; v[4] = t;
    t = v[3]; v[3] = v[6]; v[6] = t;
}
template <class R>
__device__ __forceinline__ void dft4(Cx<R>& a, Cx<R>& b, Cx<R>& c, Cx<R>& d) {
    const Cx<R> s0 = {a.re + c.re, a.im + c.im}, d0 = {a.re - c.re, a.im - c.im};
    const Cx<R> s1 = {b.re + d.re, b.im + d.im}, d1 = {b.im - d.im, d.re - b.re};  // -i (b - d)
    a = {s0.re + s1.re, s0.im + s1.im};
    b = {d0.re + d1.re, d0.im + d1.im};
    c = {s0.re - s1.re, s0.im - s1.im};
    d = {d0.re - d1.re, d0.im - d1.im};
}

// FFT of one row pair by the M/8 threads t: on entry v[q] = x[t + q M/8], on return v[q] = X[t + q M/8].
// z: the pair's padded row of shared memory; the whole block calls.
template <class R, int M, int LOGM>
__device__ __forceinline__ void fft_regs(Cx<R> (&v)[8], Cx<R>* z, int t, const Cx<R>* __restrict__ tw) {
    constexpr int T = M / 8;
    dft8(v);
    __syncthreads();  // (the row may still be read by the previous use)
#pragma unroll
    for (int q = 0; q < 8; ++q) z[dst_pad(8 * t + q)] = v[q];
    __syncthreads();
    int l = 8;
    constexpr int full = LOGM / 3, rest = LOGM % 3;  // radix-8 passes, log2 of the last radix (0: none)
#pragma unroll
    for (int p = 1; p < full; ++p) {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = z[dst_pad(t + q * T)];
        const int k = t & (l - 1), u = k * (M / (8 * l));
        const Cx<R> w1 = tw[u], w2 = tw[2 * u], w4 = tw[4 * u], w3 = cmul(w1, w2);
        v[1] = cmul(v[1], w1); v[2] = cmul(v[2], w2); v[3] = cmul(v[3], w3); v[4] = cmul(v[4], w4);
        v[5] = cmul(v[5], cmul(w1, w4)); v[6] = cmul(v[6], cmul(w2, w4)); v[7] = cmul(v[7], cmul(w3, w4));
        dft8(v);
        if (p + 1 < full || rest) {
            __syncthreads();
            const int o = (t - k) * 8 + k;
#pragma unroll
            for (int q = 0; q < 8; ++q) z[dst_pad(o + q * l)] = v[q];
            __syncthreads();
        }
        l *= 8;
    }
    if constexpr (rest == 2) {
        // radix 4, l = M/4: butterflies t and t + M/8
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = z[dst_pad(t + q * T)];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int k = t + s * T;
            const Cx<R> w1 = tw[k], w2 = tw[2 * k];
            v[s + 2] = cmul(v[s + 2], w1);
            v[s + 4] = cmul(v[s + 4], w2);
            v[s + 6] = cmul(v[s + 6], cmul(w1, w2));
            dft4(v[s], v[s + 2], v[s + 4], v[s + 6]);
        }
    } else if constexpr (rest == 1) {
        // radix 2, l = M/2: butterflies t + s M/8
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = z[dst_pad(t + q * T)];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const Cx<R> a = v[s], b = cmul(v[s + 4], tw[t + s * T]);
            v[s] = {a.re + b.re, a.im + b.im};
            v[s + 4] = {a.re - b.re, a.im - b.im};
        }
    }
}

// odd extension of the row pair (get(0 / 1, e), e in [0, n)) as complex elements t + q M/8
template <class R, int M, class Get>
__device__ __forceinline__ void load_odd(Cx<R> (&v)[8], int t, int n, Get get) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int j = t + q * (M / 8);
        if (q < 4) v[q] = j >= 1 ? Cx<R>{get(0, j - 1), get(1, j - 1)} : Cx<R>{R(0), R(0)};
        else v[q] = j > n + 1 ? Cx<R>{-get(0, M - j - 1), -get(1, M - j - 1)} : Cx<R>{R(0), R(0)};
    }
}

// The rows of a block written transposed: out[(plane n + e) rows_per_plane + row], through shared
// memory so that the block's rows of one e are written together. v[q < NQ] holds elements
// t + q M/8 - 1 of the pair f.
template <class R, int M, int NQ = 4>
__device__ __forceinline__ void store_transposed(const Cx<R> (&v)[8], Cx<R>* smem, int f, int t, int r0, int nrows, int n,
                                                 int rows_per_plane, R* __restrict__ out) {
    using C = DstCfg<M>;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int j = t + q * (M / 8);
        // DST-I of the pair: row 0 is -Im / 2, row 1 is Re / 2
        smem[(size_t)j * C::F + f] = {v[q].im * R(-0.5), v[q].re * R(0.5)};
    }
    __syncthreads();
    const R* s = reinterpret_cast<const R*>(smem);
    static_assert(C::NT % C::RB == 0, "a thread writes one row");
    const int r = threadIdx.x % C::RB, row = r0 + r;
    if (row >= nrows) return;
    const int pl = row / rows_per_plane, rr = row - pl * rows_per_plane;
    R* o = out + (size_t)pl * n * rows_per_plane + rr;
    for (int e = threadIdx.x / C::RB; e < n; e += C::NT / C::RB) o[(size_t)e * rows_per_plane] = s[(e + 1) * C::RB + r];
}

// The rows of a pair written to field component comp[k] (rows are (plane k, j) of length n)
template <class R, int M, int NQ = 4>
__device__ __forceinline__ void store_field(const Cx<R> (&v)[8], int t, int row0, int nrows, int n, int ny, R* base,
                                            size_t cstride, int pitch, int c0, int c1, int c2) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = row0 + r;
        if (row >= nrows) continue;
        const int k = row / ny, j = row - k * ny;
        R* o = base + (size_t)(k == 0 ? c0 : (k == 1 ? c1 : c2)) * cstride + (size_t)(j + kGuardAlloc) * pitch + kGuardAlloc;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int i = t + q * (M / 8);
            if (i >= 1 && i <= n) o[i - 1] = r ? v[q].re * R(0.5) : v[q].im * R(-0.5);
        }
    }
}

// Pass over rows: DST-I of every row of length n, written transposed:
// out[(row / rows_per_plane) * n * rows_per_plane + e * rows_per_plane + row % rows_per_plane]
template <class R, int M, int LOGM>
__global__ void __launch_bounds__(DstCfg<M>::NT, 1024 / DstCfg<M>::NT) k_dst_pass_t(const R* __restrict__ in, int nrows, int n,
                                                              int rows_per_plane, R* __restrict__ out,
                                                              const Cx<R>* __restrict__ tw) {
    HPQ_PDL_ENTRY();
    using C = DstCfg<M>;
    extern __shared__ __align__(16) unsigned char dst_smem[];
    Cx<R>* z = reinterpret_cast<Cx<R>*>(dst_smem);
    const int f = threadIdx.x / C::T, t = threadIdx.x % C::T, r0 = blockIdx.x * C::RB, row0 = r0 + 2 * f;
    auto get = [&](int r, int e) -> R { return row0 + r < nrows ? in[(size_t)(row0 + r) * n + e] : R(0); };
    Cx<R> v[8];
    load_odd<R, M>(v, t, n, get);
    fft_regs<R, M, LOGM>(v, z + f * C::MP, t, tw);
    store_transposed<R, M>(v, z, f, t, r0, nrows, n, rows_per_plane, out);
}

// y-pass, eigenvalue multiply, y-pass; rows are (plane, i) of length n = ny; eig is [j][i] with
// row length rows_per_plane; written transposed back to [plane][j][i]
template <class R, int M, int LOGM, class Eig>
__device__ __forceinline__ void dst_pass_eig(const R* __restrict__ in, int nrows, int n, int rows_per_plane, Eig eig,
                                             R* __restrict__ out, const Cx<R>* __restrict__ tw) {
    using C = DstCfg<M>;
    extern __shared__ __align__(16) unsigned char dst_smem[];
    Cx<R>* z = reinterpret_cast<Cx<R>*>(dst_smem);
    const int f = threadIdx.x / C::T, t = threadIdx.x % C::T, r0 = blockIdx.x * C::RB, row0 = r0 + 2 * f;
    auto get = [&](int r, int e) -> R { return row0 + r < nrows ? in[(size_t)(row0 + r) * n + e] : R(0); };
    Cx<R> v[8];
    load_odd<R, M>(v, t, n, get);
    Cx<R>* zf = z + f * C::MP;
    fft_regs<R, M, LOGM>(v, zf, t, tw);
    // odd extension of the products; elements beyond M/2 are those of the mirrored thread
    const int i0 = row0 % rows_per_plane, i1 = (row0 + 1) % rows_per_plane;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int j = t + q * (M / 8);
        Cx<R> w{R(0), R(0)};
        if (j >= 1) {
            w.re = row0 < nrows ? v[q].im * R(-0.5) * eig(j - 1, i0) : R(0);
            w.im = row0 + 1 < nrows ? v[q].re * R(0.5) * eig(j - 1, i1) : R(0);
        }
        v[q] = w;
        zf[j] = w;
    }
    __syncthreads();
#pragma unroll
    for (int q = 4; q < 8; ++q) {
        const int j = t + q * (M / 8);
        const Cx<R> w = j > M / 2 ? zf[M - j] : Cx<R>{R(0), R(0)};
        v[q] = {-w.re, -w.im};
    }
    // (the twiddles are read again: kept over the first transform they cost 60 registers in double)
    asm volatile("" : "+l"(tw));
    fft_regs<R, M, LOGM>(v, zf, t, tw);
    store_transposed<R, M>(v, z, f, t, r0, nrows, n, rows_per_plane, out);
}
template <class R, int M, int LOGM>
__global__ void __launch_bounds__(DstCfg<M>::NT, 1024 / DstCfg<M>::NT) k_dst_pass_eig(const R* __restrict__ in, int nrows, int n,
                                                                int rows_per_plane, const R* __restrict__ eig,
                                                                R* __restrict__ out, const Cx<R>* __restrict__ tw) {
    HPQ_PDL_ENTRY();
    dst_pass_eig<R, M, LOGM>(in, nrows, n, rows_per_plane,
                             [&](int e, int i) { return eig[(size_t)e * rows_per_plane + i]; }, out, tw);
}

// final x-pass: rows are (plane k, j) of length nx; result scattered into field component comp[k]
template <class R, int M, int LOGM>
__global__ void __launch_bounds__(DstCfg<M>::NT, 1024 / DstCfg<M>::NT) k_dst_pass_field(const R* __restrict__ in, int nrows, int n, int ny,
                                                                  R* base, size_t cstride, int pitch, int c0, int c1,
                                                                  int c2, const Cx<R>* __restrict__ tw) {
    HPQ_PDL_ENTRY();
    using C = DstCfg<M>;
    extern __shared__ __align__(16) unsigned char dst_smem[];
    Cx<R>* z = reinterpret_cast<Cx<R>*>(dst_smem);
    const int f = threadIdx.x / C::T, t = threadIdx.x % C::T, row0 = blockIdx.x * C::RB + 2 * f;
    auto get = [&](int r, int e) -> R { return row0 + r < nrows ? in[(size_t)(row0 + r) * n + e] : R(0); };
    Cx<R> v[8];
    load_odd<R, M>(v, t, n, get);
    fft_regs<R, M, LOGM>(v, z + f * C::MP, t, tw);
    store_field<R, M>(v, t, row0, nrows, n, ny, base, cstride, pitch, c0, c1, c2);
}

// ------------------------------------------------------------------------------------------
// Any length: Bluestein's chirp-z algorithm (L. Bluestein, "A linear filtering approach to the
// computation of the discrete Fourier transform", 1970). With d_m = exp(-i pi m^2 / M), the DFT of
// the odd extension z (length M = 2(n+1), not a power of two) is
//   Z[k] = d_k sum_j (z_j d_j) conj(d_{k-j}),
// a circular convolution of length L (a power of two >= 2M - 1) done with two FFTs of length L: the
// forward one, the product with B = FFT(conj(d)), and the inverse through conj(FFT(conj(.))). The FFTs
// are the register FFT above; z fills less than half of L, and Z is needed in less than a quarter.
// ------------------------------------------------------------------------------------------
template <class R>
struct BluAxis {
    const Cx<R>* d;    // chirp d_m, m < M
    const Cx<R>* B;    // FFT_L of the chirp filter conj(d_|m|), divided by L
    const Cx<R>* tw;   // exp(-2 pi i t / L), t < L/2
    int M;
};

// DST-I of one row pair by the L/8 threads t: on return v[q], q < 2, holds {row 1, -row 0} times 2 at
// element t + q L/8 - 1, as the power-of-two transform leaves it
template <class R, int L, int LOGL, class Get>
__device__ __forceinline__ void blu_rows(Cx<R> (&v)[8], Cx<R>* z, int t, int n, const BluAxis<R>& A, Get get) {
    const int M = A.M;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int j = t + q * (L / 8);
        v[q] = {R(0), R(0)};
        if (q < 4 && j >= 1 && j < M && j != n + 1) {
            const bool up = j <= n;
            const int e = up ? j - 1 : M - j - 1;
            const R sg = up ? R(1) : R(-1);
            v[q] = cmul(Cx<R>{sg * get(0, e), sg * get(1, e)}, A.d[j]);
        }
    }
    const Cx<R>* tw = A.tw;
    fft_regs<R, L, LOGL>(v, z, t, tw);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const Cx<R> p = cmul(v[q], A.B[t + q * (L / 8)]);
        v[q] = {p.re, -p.im};
    }
    asm volatile("" : "+l"(tw));  // (read again rather than kept)
    fft_regs<R, L, LOGL>(v, z, t, tw);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int k = t + q * (L / 8);
        if (k < M) v[q] = cmul(Cx<R>{v[q].re, -v[q].im}, A.d[k]);
    }
}

template <class R, int L, int LOGL>
__global__ void __launch_bounds__(DstCfg<L>::NT, 1024 / DstCfg<L>::NT) k_dstb_pass_t(const R* __restrict__ in, int nrows,
                                                                                     int n, int rows_per_plane,
                                                                                     R* __restrict__ out, BluAxis<R> A) {
    HPQ_PDL_ENTRY();
    using C = DstCfg<L>;
    extern __shared__ __align__(16) unsigned char dst_smem[];
    Cx<R>* z = reinterpret_cast<Cx<R>*>(dst_smem);
    const int f = threadIdx.x / C::T, t = threadIdx.x % C::T, r0 = blockIdx.x * C::RB, row0 = r0 + 2 * f;
    auto get = [&](int r, int e) -> R { return row0 + r < nrows ? in[(size_t)(row0 + r) * n + e] : R(0); };
    Cx<R> v[8];
    blu_rows<R, L, LOGL>(v, z + f * C::MP, t, n, A, get);
    store_transposed<R, L, 2>(v, z, f, t, r0, nrows, n, rows_per_plane, out);
}

template <class R, int L, int LOGL>
__global__ void __launch_bounds__(DstCfg<L>::NT, 1024 / DstCfg<L>::NT) k_dstb_pass_eig(const R* __restrict__ in, int nrows,
                                                                                       int n, int rows_per_plane,
                                                                                       const R* __restrict__ eig,
                                                                                       R* __restrict__ out, BluAxis<R> A) {
    HPQ_PDL_ENTRY();
    using C = DstCfg<L>;
    extern __shared__ __align__(16) unsigned char dst_smem[];
    Cx<R>* z = reinterpret_cast<Cx<R>*>(dst_smem);
    const int f = threadIdx.x / C::T, t = threadIdx.x % C::T, r0 = blockIdx.x * C::RB, row0 = r0 + 2 * f;
    auto get = [&](int r, int e) -> R { return row0 + r < nrows ? in[(size_t)(row0 + r) * n + e] : R(0); };
    Cx<R> v[8];
    Cx<R>* zf = z + f * C::MP;
    blu_rows<R, L, LOGL>(v, zf, t, n, A, get);
    const int i0 = row0 % rows_per_plane, i1 = (row0 + 1) % rows_per_plane;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int j = t + q * (L / 8);
        if (j >= 1 && j <= n) {
            const R* eg = eig + (size_t)(j - 1) * rows_per_plane;
            zf[j - 1] = {row0 < nrows ? v[q].im * R(-0.5) * eg[i0] : R(0), row0 + 1 < nrows ? v[q].re * R(0.5) * eg[i1] : R(0)};
        }
    }
    __syncthreads();
    auto get2 = [&](int r, int e) -> R { return r ? zf[e].im : zf[e].re; };
    blu_rows<R, L, LOGL>(v, zf, t, n, A, get2);
    store_transposed<R, L, 2>(v, z, f, t, r0, nrows, n, rows_per_plane, out);
}

template <class R, int L, int LOGL>
__global__ void __launch_bounds__(DstCfg<L>::NT, 1024 / DstCfg<L>::NT)
    k_dstb_pass_field(const R* __restrict__ in, int nrows, int n, int ny, R* base, size_t cstride, int pitch, int c0, int c1,
                      int c2, BluAxis<R> A) {
    HPQ_PDL_ENTRY();
    using C = DstCfg<L>;
    extern __shared__ __align__(16) unsigned char dst_smem[];
    Cx<R>* z = reinterpret_cast<Cx<R>*>(dst_smem);
    const int f = threadIdx.x / C::T, t = threadIdx.x % C::T, row0 = blockIdx.x * C::RB + 2 * f;
    auto get = [&](int r, int e) -> R { return row0 + r < nrows ? in[(size_t)(row0 + r) * n + e] : R(0); };
    Cx<R> v[8];
    blu_rows<R, L, LOGL>(v, z + f * C::MP, t, n, A, get);
    store_field<R, L, 2>(v, t, row0, nrows, n, ny, base, cstride, pitch, c0, c1, c2);
}

template <class R>
class FastDST {
public:
    int nx = 0, ny = 0, Mx = 0, My = 0;  // radix-2 lengths 2(n+1), or 0 on a Bluestein axis
    int Lx = 0, Ly = 0;                  // Bluestein lengths, or 0 on a radix-2 axis
    Cx<R>* twx = nullptr;
    Cx<R>* twy = nullptr;
    BluAxis<R> bx{}, by{};

    static int pow2_len(int n) {
        const int m = 2 * (n + 1);
        return (m >= 64 && m <= 4096 && (m & (m - 1)) == 0) ? m : 0;
    }
    // Bluestein convolution length: the smallest power of two >= 2M - 1, M = 2(n+1); up to n = 2047
    static int blu_len(int n) {
        if (n < 1) return 0;
        const int m = 2 * (n + 1);
        int l = 64;
        while (l < 2 * m - 1) l <<= 1;
        return l <= 8192 ? l : 0;
    }
    static bool axis_ok(int n) { return pow2_len(n) || blu_len(n); }
    static bool supported(int nx, int ny) { return axis_ok(nx) && axis_ok(ny); }
    static bool radix2(int nx, int ny) { return pow2_len(nx) && pow2_len(ny); }

    // chirp, filter spectrum (natural order, divided by L) and twiddles of a Bluestein axis, from FP64 tables
    static BluAxis<R> blu_axis(int n, int L) {
        const int M = 2 * (n + 1);
        const double pi = 3.14159265358979323846;
        std::vector<double> dre(M), dim(M);
        for (int m = 0; m < M; ++m) {
            const long long q = ((long long)m * m) % (2LL * M);  // d_m = exp(-i pi m^2 / M), m^2 mod 2M exact
            dre[m] = std::cos(pi * (double)q / M);
            dim[m] = -std::sin(pi * (double)q / M);
        }
        // b_m = conj(d_|m|) on the circle of length L, then its DFT (iterative radix 2, FP64)
        std::vector<double> br(L, 0.0), bi(L, 0.0);
        for (int m = 0; m < M; ++m) { br[m] = dre[m]; bi[m] = -dim[m]; }
        for (int m = 1; m < M; ++m) { br[L - m] = dre[m]; bi[L - m] = -dim[m]; }
        int logl = 0;
        while ((1 << logl) < L) ++logl;
        auto rev = [&](int j) {
            int r = 0;
            for (int b = 0; b < logl; ++b) r |= ((j >> b) & 1) << (logl - 1 - b);
            return r;
        };
        for (int j = 0; j < L; ++j) {
            const int r = rev(j);
            if (r > j) { std::swap(br[j], br[r]); std::swap(bi[j], bi[r]); }
        }
        for (int len = 2; len <= L; len <<= 1)
            for (int i0 = 0; i0 < L; i0 += len)
                for (int k = 0; k < len / 2; ++k) {
                    const double c = std::cos(2 * pi * k / len), sn = -std::sin(2 * pi * k / len);
                    const int a = i0 + k, b = a + len / 2;
                    const double vr = br[b] * c - bi[b] * sn, vi = br[b] * sn + bi[b] * c;
                    br[b] = br[a] - vr; bi[b] = bi[a] - vi;
                    br[a] += vr; bi[a] += vi;
                }
        std::vector<Cx<R>> hd(M), hB(L);
        for (int m = 0; m < M; ++m) hd[m] = {(R)dre[m], (R)dim[m]};
        for (int q = 0; q < L; ++q) hB[q] = {(R)(br[q] / L), (R)(bi[q] / L)};
        BluAxis<R> A{};
        Cx<R>*d = nullptr, *B = nullptr;
        HPQ_CUDA(cudaMalloc(&d, M * sizeof(Cx<R>)));
        HPQ_CUDA(cudaMalloc(&B, L * sizeof(Cx<R>)));
        HPQ_CUDA(cudaMemcpy(d, hd.data(), M * sizeof(Cx<R>), cudaMemcpyHostToDevice));
        HPQ_CUDA(cudaMemcpy(B, hB.data(), L * sizeof(Cx<R>), cudaMemcpyHostToDevice));
        A.d = d;
        A.B = B;
        A.tw = twiddles(L);
        A.M = M;
        return A;
    }
    static void free_axis(BluAxis<R>& A) {
        if (A.d) cudaFree(const_cast<Cx<R>*>(A.d));
        if (A.B) cudaFree(const_cast<Cx<R>*>(A.B));
        if (A.tw) cudaFree(const_cast<Cx<R>*>(A.tw));
        A = BluAxis<R>{};
    }

    static Cx<R>* twiddles(int M) {
        std::vector<Cx<R>> h(M / 2);
        const double pi = 3.14159265358979323846;
        for (int k = 0; k < M / 2; ++k) h[k] = {(R)std::cos(2 * pi * k / M), (R)(-std::sin(2 * pi * k / M))};
        Cx<R>* d;
        HPQ_CUDA(cudaMalloc(&d, h.size() * sizeof(Cx<R>)));
        HPQ_CUDA(cudaMemcpy(d, h.data(), h.size() * sizeof(Cx<R>), cudaMemcpyHostToDevice));
        return d;
    }
    void init(int nx_, int ny_) {
        nx = nx_; ny = ny_;
        Mx = pow2_len(nx); My = pow2_len(ny);
        Lx = Mx ? 0 : blu_len(nx);
        Ly = My ? 0 : blu_len(ny);
        if (!(Mx || Lx) || !(My || Ly)) throw CudaError("FastDST: grid too large for the FFT DST");
        if (Mx) twx = twiddles(Mx); else bx = blu_axis(nx, Lx);
        if (My) twy = twiddles(My); else by = blu_axis(ny, Ly);
        set_attrs<64, 6>(); set_attrs<128, 7>(); set_attrs<256, 8>(); set_attrs<512, 9>();
        set_attrs<1024, 10>(); set_attrs<2048, 11>(); set_attrs<4096, 12>();
        if (Lx || Ly) {
            set_attrs_blu<64, 6>(); set_attrs_blu<128, 7>(); set_attrs_blu<256, 8>(); set_attrs_blu<512, 9>();
            set_attrs_blu<1024, 10>(); set_attrs_blu<2048, 11>(); set_attrs_blu<4096, 12>(); set_attrs_blu<8192, 13>();
        }
    }
    void release() {
        if (twx) cudaFree(twx);
        if (twy) cudaFree(twy);
        twx = twy = nullptr;
        free_axis(bx);
        free_axis(by);
    }
    template <int L, int LOGL>
    static void set_attrs_blu() {
        const int smem = (int)DstCfg<L>::template smem<R>();
        HPQ_CUDA(cudaFuncSetAttribute(k_dstb_pass_t<R, L, LOGL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        HPQ_CUDA(cudaFuncSetAttribute(k_dstb_pass_eig<R, L, LOGL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        HPQ_CUDA(cudaFuncSetAttribute(k_dstb_pass_field<R, L, LOGL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    }
    template <int L, int LOGL>
    void bpass_t(cudaStream_t st, const R* in, int nrows, int n, int rpp, R* out, const BluAxis<R>& A) {
        using C = DstCfg<L>;
        hpq_launch(k_dstb_pass_t<R, L, LOGL>, dst_grid<L>(nrows), dim3(C::NT), C::template smem<R>(), st, in, nrows, n, rpp, out, A);
        HPQ_LAUNCH_CHECK();
    }
    template <int L, int LOGL>
    void bpass_eig(cudaStream_t st, const R* in, int nrows, int n, int rpp, const R* eig, R* out, const BluAxis<R>& A) {
        using C = DstCfg<L>;
        hpq_launch(k_dstb_pass_eig<R, L, LOGL>, dst_grid<L>(nrows), dim3(C::NT), C::template smem<R>(), st, in, nrows, n, rpp, eig, out, A);
        HPQ_LAUNCH_CHECK();
    }
    template <int L, int LOGL>
    void bpass_field(cudaStream_t st, const R* in, int nrows, int n, R* base, size_t cs, int pitch, const int* comps,
                     int nrhs, const BluAxis<R>& A) {
        using C = DstCfg<L>;
        hpq_launch(k_dstb_pass_field<R, L, LOGL>, dst_grid<L>(nrows), dim3(C::NT), C::template smem<R>(), st,
                   in, nrows, n, ny, base, cs, pitch, comps[0], nrhs > 1 ? comps[1] : comps[0],
                   nrhs > 2 ? comps[2] : comps[0], A);
        HPQ_LAUNCH_CHECK();
    }
    template <int M, int LOGM>
    static void set_attrs() {
        const int smem = (int)DstCfg<M>::template smem<R>();
        HPQ_CUDA(cudaFuncSetAttribute(k_dst_pass_t<R, M, LOGM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        HPQ_CUDA(cudaFuncSetAttribute(k_dst_pass_eig<R, M, LOGM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        HPQ_CUDA(cudaFuncSetAttribute(k_dst_pass_field<R, M, LOGM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    }
    template <int M>
    static dim3 dst_grid(int nrows) { return dim3((nrows + DstCfg<M>::RB - 1) / DstCfg<M>::RB); }
    template <int M, int LOGM>
    void pass_t(cudaStream_t st, const R* in, int nrows, int n, int rpp, R* out, const Cx<R>* tw) {
        using C = DstCfg<M>;
        hpq_launch(k_dst_pass_t<R, M, LOGM>, dst_grid<M>(nrows), dim3(C::NT), C::template smem<R>(), st, in, nrows, n, rpp, out, tw);
        HPQ_LAUNCH_CHECK();
    }
    template <int M, int LOGM>
    void pass_eig(cudaStream_t st, const R* in, int nrows, int n, int rpp, const R* eig, R* out, const Cx<R>* tw) {
        using C = DstCfg<M>;
        hpq_launch(k_dst_pass_eig<R, M, LOGM>, dst_grid<M>(nrows), dim3(C::NT), C::template smem<R>(), st, in, nrows, n, rpp, eig, out, tw);
        HPQ_LAUNCH_CHECK();
    }
    template <int M, int LOGM>
    void pass_field(cudaStream_t st, const R* in, int nrows, int n, R* base, size_t cs, int pitch, const int* comps,
                    int nrhs, const Cx<R>* tw) {
        using C = DstCfg<M>;
        hpq_launch(k_dst_pass_field<R, M, LOGM>, dst_grid<M>(nrows), dim3(C::NT), C::template smem<R>(), st,
            in, nrows, n, ny, base, cs, pitch, comps[0], nrhs > 1 ? comps[1] : comps[0], nrhs > 2 ? comps[2] : comps[0], tw);
        HPQ_LAUNCH_CHECK();
    }

#define HPQ_DST_DISPATCH(Mval, CALL)                       \
    switch (Mval) {                                        \
        case 64: CALL(64, 6); break;                       \
        case 128: CALL(128, 7); break;                     \
        case 256: CALL(256, 8); break;                     \
        case 512: CALL(512, 9); break;                     \
        case 1024: CALL(1024, 10); break;                  \
        case 2048: CALL(2048, 11); break;                  \
        case 4096: CALL(4096, 12); break;                  \
        default: throw CudaError("unsupported DST length"); \
    }

#define HPQ_DSTB_DISPATCH(Lval, CALL)                      \
    switch (Lval) {                                        \
        case 64: CALL(64, 6); break;                       \
        case 128: CALL(128, 7); break;                     \
        case 256: CALL(256, 8); break;                     \
        case 512: CALL(512, 9); break;                     \
        case 1024: CALL(1024, 10); break;                  \
        case 2048: CALL(2048, 11); break;                  \
        case 4096: CALL(4096, 12); break;                  \
        case 8192: CALL(8192, 13); break;                  \
        default: throw CudaError("unsupported Bluestein length"); \
    }

    // stage: nrhs planes [k][j][i] (nx contiguous); work: scratch of the same size; eig [j][i]
    void solve(cudaStream_t st, int nrhs, R* stage, R* work, const R* eig, R* base, size_t cs, int pitch,
               const int* comps) {
        if (Mx) {
#define CALL1(M, L) pass_t<M, L>(st, stage, nrhs * ny, nx, ny, work, twx)
            HPQ_DST_DISPATCH(Mx, CALL1)
#undef CALL1
        } else {
#define CALL1(L, G) bpass_t<L, G>(st, stage, nrhs * ny, nx, ny, work, bx)
            HPQ_DSTB_DISPATCH(Lx, CALL1)
#undef CALL1
        }
        if (My) {
#define CALL2(M, L) pass_eig<M, L>(st, work, nrhs * nx, ny, nx, eig, stage, twy)
            HPQ_DST_DISPATCH(My, CALL2)
#undef CALL2
        } else {
#define CALL2(L, G) bpass_eig<L, G>(st, work, nrhs * nx, ny, nx, eig, stage, by)
            HPQ_DSTB_DISPATCH(Ly, CALL2)
#undef CALL2
        }
        if (Mx) {
#define CALL3(M, L) pass_field<M, L>(st, stage, nrhs * ny, nx, base, cs, pitch, comps, nrhs, twx)
            HPQ_DST_DISPATCH(Mx, CALL3)
#undef CALL3
        } else {
#define CALL3(L, G) bpass_field<L, G>(st, stage, nrhs * ny, nx, base, cs, pitch, comps, nrhs, bx)
            HPQ_DSTB_DISPATCH(Lx, CALL3)
#undef CALL3
        }
    }
};

}  // namespace hpq

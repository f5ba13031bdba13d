// Allocation-free Dirichlet Poisson solve (hpq_poisson_dirichlet_noalloc in include/hpq.h).
//
// Some callers of this library cannot call cudaMalloc: code that runs while a CUDA stream is
// being captured into a graph (allocation is not a capturable operation), plugins of host
// frameworks that own the device memory pool and forbid side allocations, and real-time loops
// that must not pay for or fail on an allocation at solve time. This entry point serves them:
// the caller passes the right-hand side and the solution buffer; the transformed intermediate of
// the solve lives in one file-scope device array of fixed size (the FFT twiddles of every length are
// constant data beside it; the eigenvalues are formed where they are used). CUDA loads the
// library's device code lazily, so the array's
// memory is committed on a device by the first call on that device (which can therefore fail
// with HPQ_ERR_CUDA when the device is already full) and held until the process exits.
//
// Limit: nx and ny of the form 2^k - 1 with 31 <= n <= 1023 (the shared-memory FFT path of the
// DST-I), i.e. at most 1023 x 1023 cells; the scratch array is 8.0 MiB.
// All calls share the array and it keeps the contents of the last call. Every element a solve
// reads is written earlier in the same solve, so nothing needs clearing between calls; two
// calls whose kernels overlap on the GPU (different streams, or different host threads on one
// stream without ordering) race on the array and give wrong results.
// Errors: a CUDA error already pending when the call starts is left to the caller (the call
// returns HPQ_ERR_CUDA without launching or clearing it); each launch is checked right after it
// is made.
#include <cuda_runtime.h>

#include <mutex>

#include "../../include/hpq.h"
#include "fftdst.cuh"

namespace {

constexpr int kMaxN = 1023;
constexpr size_t kPlane = (size_t)kMaxN * kMaxN;          // one nx x ny plane
constexpr size_t kTw = 2016;                               // complex twiddles of M = 64 .. 2048, M/2 each

static __device__ __align__(256) double g_poisson_scratch[kPlane];  // work plane
// Twiddles exp(-2 pi i k / M), k < M/2, of M = 64 .. 2048 in this order, as constant data of the
// library's device code: they are there whichever stream or capture makes the first call. Formed by
// the compiler: the Taylor series of sine and cosine on [0, pi/4] in pairs of doubles (Dekker, "A
// floating-point technique for extending the available precision", 1971), then symmetry.
struct Pair {
    double hi, lo;
};
constexpr Pair two_sum(double a, double b) {
    const double s = a + b, t = s - a;
    return {s, (a - (s - t)) + (b - t)};
}
constexpr Pair two_mul(double a, double b) {
    const double c = 134217729.0;  // 2^27 + 1
    const double ah = c * a - (c * a - a), al = a - ah, bh = c * b - (c * b - b), bl = b - bh, p = a * b;
    return {p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr Pair add(Pair a, Pair b) {
    const Pair s = two_sum(a.hi, b.hi);
    return two_sum(s.hi, s.lo + a.lo + b.lo);
}
constexpr Pair mul(Pair a, Pair b) {
    const Pair p = two_mul(a.hi, b.hi);
    return two_sum(p.hi, p.lo + (a.hi * b.lo + a.lo * b.hi));
}
constexpr Pair over(Pair a, double n) {  // a / n
    const double q = a.hi / n;
    const Pair p = two_mul(q, n);
    return two_sum(q, (((a.hi - p.hi) - p.lo) + a.lo) / n);
}
struct Twiddles {
    double v[2 * kTw];
};
constexpr size_t tw_offset(int M) { return (size_t)M / 2 - 32; }  // 32 + 64 + .. + M/4 before length M
constexpr Twiddles make_twiddles() {
    Twiddles t{};
    double c[257] = {}, s[257] = {};  // cos, sin of 2 pi k / 2048 in the first octant
    for (int k = 0; k <= 256; ++k) {
        const Pair x = mul({3.14159265358979323846, 1.2246467991473532e-16}, {k / 1024.0, 0.0}), x2 = mul(x, x);
        Pair p{1.0, 0.0}, q = x, sc{0.0, 0.0}, ss{0.0, 0.0};
        for (int n = 0; n < 12; ++n) {  // terms 2n and 2n + 1; the first one left out is below 1e-26
            sc = add(sc, p);
            ss = add(ss, q);
            p = over(mul(p, x2), -(2.0 * n + 1) * (2 * n + 2));
            q = over(mul(q, x2), -(2.0 * n + 2) * (2 * n + 3));
        }
        c[k] = sc.hi;
        s[k] = ss.hi;
    }
    for (int M = 64; M <= 2048; M *= 2)
        for (int k = 0; k < M / 2; ++k) {
            const int a = k * (2048 / M), h = a <= 512 ? a : 1024 - a;  // angle, folded into the first quarter
            const double co = h <= 256 ? c[h] : s[512 - h], si = h <= 256 ? s[h] : c[512 - h];
            t.v[2 * (tw_offset(M) + k)] = a <= 512 ? co : -co;
            t.v[2 * (tw_offset(M) + k) + 1] = -si;
        }
    return t;
}
static __device__ __align__(256) const Twiddles g_poisson_twiddles = make_twiddles();

constexpr int kMaxDevices = 64;
std::mutex g_mutex;
double* g_scratch_ptr[kMaxDevices] = {};
const hpq::Cx<double>* g_twiddle_ptr[kMaxDevices] = {};

cudaError_t set_smem_attributes();

// Set-up, once per device with that device current: the host addresses of the arrays are only
// stand-ins, kernels must be given the device addresses returned here. The shared-memory limits of
// the pass kernels are raised at the same time, so later calls make no set-up call at all. Nothing
// is copied or launched, so that no stream has to wait for it.
int scratch_for_current_device(double** out, const hpq::Cx<double>** tw) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return HPQ_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_poisson_scratch) != cudaSuccess || !p) return HPQ_ERR_CUDA;
        if (set_smem_attributes() != cudaSuccess) return HPQ_ERR_CUDA;
        void* t = nullptr;
        if (cudaGetSymbolAddress(&t, g_poisson_twiddles) != cudaSuccess || !t) return HPQ_ERR_CUDA;
        g_twiddle_ptr[dev] = static_cast<const hpq::Cx<double>*>(t);
        g_scratch_ptr[dev] = static_cast<double*>(p);
    }
    *out = g_scratch_ptr[dev];
    *tw = g_twiddle_ptr[dev];
    return HPQ_OK;
}

// y-pass, division by the eigenvalues of the 5-point Laplacian (with the normalisation of the two
// DST-I per axis), y-pass. The eigenvalues are separable: a thread needs the sines of its two rows and
// four columns, where a table of nx * ny took a kernel of its own and two sines per point.
template <int M, int LOGM>
__global__ void __launch_bounds__(hpq::DstCfg<M>::NT, 1024 / hpq::DstCfg<M>::NT) k_pass_eig(const double* __restrict__ in, int nx, int ny, double dx,
                                                                 double dy, double* __restrict__ out,
                                                                 const hpq::Cx<double>* __restrict__ tw) {
    HPQ_PDL_ENTRY();
    const double norm = (2.0 / (nx + 1)) * (2.0 / (ny + 1));
    auto lambda = [](int k, int n, double h) {
        const double s = sinpi((k + 1) / (2.0 * (n + 1)));
        return s * s / (h * h);
    };
    hpq::dst_pass_eig<double, M, LOGM>(
        in, nx, ny, nx, [&](int e, int i) { return norm / (-4.0 * (lambda(i, nx, dx) + lambda(e, ny, dy))); }, out, tw);
}

template <int M, int LOGM>
cudaError_t set_attrs_for() {
    const int smem = (int)hpq::DstCfg<M>::template smem<double>();
    cudaError_t e = cudaFuncSetAttribute(hpq::k_dst_pass_t<double, M, LOGM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_pass_eig<M, LOGM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(hpq::k_dst_pass_field<double, M, LOGM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e;
}

cudaError_t set_smem_attributes() {
    cudaError_t e = set_attrs_for<64, 6>();
    if (e == cudaSuccess) e = set_attrs_for<128, 7>();
    if (e == cudaSuccess) e = set_attrs_for<256, 8>();
    if (e == cudaSuccess) e = set_attrs_for<512, 9>();
    if (e == cudaSuccess) e = set_attrs_for<1024, 10>();
    if (e == cudaSuccess) e = set_attrs_for<2048, 11>();
    return e;
}

// Launch of one pass; a dependent one may start before the pass in front of it has ended (its
// prologue waits for that pass)
template <int M, class... K, class... A>
cudaError_t launch(void (*kernel)(K...), cudaStream_t st, int nrows, bool dependent, A... args) {
    using C = hpq::DstCfg<M>;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((nrows + C::RB - 1) / C::RB);
    cfg.blockDim = dim3(C::NT);
    cfg.dynamicSmemBytes = C::template smem<double>();
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = dependent && hpq::pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int M, int LOGM>
cudaError_t pass_t(cudaStream_t st, const double* in, int nrows, int n, int rpp, double* out,
                   const hpq::Cx<double>* tw) {
    return launch<M>(hpq::k_dst_pass_t<double, M, LOGM>, st, nrows, false, in, nrows, n, rpp, out, tw);
}
template <int M, int LOGM>
cudaError_t pass_eig(cudaStream_t st, const double* in, int nx, int ny, double dx, double dy, double* out,
                     const hpq::Cx<double>* tw) {
    return launch<M>(k_pass_eig<M, LOGM>, st, nx, true, in, nx, ny, dx, dy, out, tw);
}
// The last x-pass writes a plain nx x ny plane (the caller's solution buffer): a slab view with
// no guard cells, i.e. pitch nx and the guard offset removed from the base pointer.
template <int M, int LOGM>
cudaError_t pass_plane(cudaStream_t st, const double* in, int nrows, int n, int ny, double* out,
                       const hpq::Cx<double>* tw) {
    const int G = hpq::kGuardAlloc;
    double* base = out - ((ptrdiff_t)G * n + G);  // element (i, j) -> out[j * n + i]
    return launch<M>(hpq::k_dst_pass_field<double, M, LOGM>, st, nrows, true, in, nrows, n, ny, base, (size_t)0, n, 0, 0, 0, tw);
}

int pow2_len(int n) {
    const int m = 2 * (n + 1);
    return (n >= 31 && n <= kMaxN && (m & (m - 1)) == 0) ? m : 0;
}

#define HPQ_NOALLOC_DISPATCH(Mval, CALL) \
    switch (Mval) {                      \
        case 64: e = CALL(64, 6); break;   \
        case 128: e = CALL(128, 7); break; \
        case 256: e = CALL(256, 8); break; \
        case 512: e = CALL(512, 9); break; \
        case 1024: e = CALL(1024, 10); break; \
        case 2048: e = CALL(2048, 11); break; \
        default: return HPQ_ERR_ARG;     \
    }

}  // namespace

extern "C" int hpq_poisson_dirichlet_noalloc(const double* f, double* u, int nx, int ny, double dx, double dy,
                                             void* stream) {
    if (!f || !u || !(dx > 0) || !(dy > 0)) return HPQ_ERR_ARG;
    if (nx > kMaxN || ny > kMaxN) return HPQ_ERR_TOO_LARGE;
    const int Mx = pow2_len(nx), My = pow2_len(ny);
    if (!Mx || !My) return HPQ_ERR_ARG;
    // an error left pending by the caller's earlier work stays the caller's: nothing is launched
    // and it is not cleared
    if (cudaPeekAtLastError() != cudaSuccess) return HPQ_ERR_CUDA;
    double* work = nullptr;  // y-transformed intermediate, nx*ny
    const hpq::Cx<double>* tw = nullptr;
    if (int r = scratch_for_current_device(&work, &tw)) return r;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const auto *twx = tw + tw_offset(Mx), *twy = tw + tw_offset(My);
    cudaError_t e = cudaSuccess;
    // x-pass of f -> u (transposed, u serves as the temporary); y-pass * eig * y-pass of u ->
    // work; x-pass of work -> u. No pass reads and writes the same buffer.
#define CALL1(M, L) pass_t<M, L>(st, f, ny, nx, ny, u, twx)
    HPQ_NOALLOC_DISPATCH(Mx, CALL1)
#undef CALL1
    if (e != cudaSuccess) return HPQ_ERR_CUDA;
#define CALL2(M, L) pass_eig<M, L>(st, u, nx, ny, dx, dy, work, twy)
    HPQ_NOALLOC_DISPATCH(My, CALL2)
#undef CALL2
    if (e != cudaSuccess) return HPQ_ERR_CUDA;
#define CALL3(M, L) pass_plane<M, L>(st, work, ny, nx, ny, u, twx)
    HPQ_NOALLOC_DISPATCH(Mx, CALL3)
#undef CALL3
    if (e != cudaSuccess) return HPQ_ERR_CUDA;
    return HPQ_OK;
}

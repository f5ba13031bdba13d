// Cluster-resident multigrid: the whole solve of k_mg_solve (mg.cuh) for grids whose hierarchy fits
// the shared memory of one thread-block cluster per component.
//
// What bounds the solve at 255^2 and below is the latency between its sweeps, not bandwidth: the
// tile form of k_mg_solve passes 7 grid barriers per V-cycle and reloads every tile from L2 in each
// phase. Here each component (Bx, By: they share the operator and meet only in the norm) belongs
// to one cluster of up to 16 blocks. The rows of a level are split over the blocks, every level's
// solution, right-hand side, coefficient and inverse diagonal stay in shared memory for the whole
// solve, and after a colour sweep a block sends the boundary row it updated into its neighbours'
// halo rows (st.async to distributed shared memory, counted by an mbarrier of the receiver; a
// cluster barrier after every sweep took 1000 cycles). Levels too small to split run in block 0 of
// the cluster, with only as many warps as they have points for. The same sweeps in the same order
// as k_mg_solve.
//
// Half of the work around the sweeps falls away because a colour sweep reads the other colour
// only: of an initial guess or an interpolated correction the first sweep needs colour 1 alone (and
// nothing of a zero guess), and after the last sweep the residual of colour 1 is zero up to
// rounding, so that the restriction and the norm take colour 0.
//
// A thread owns column pairs (2k, 2k+1) of RT consecutive rows: a sweep updates one point of each
// pair. Values are held in registers by colour e = (row + column) & 1, so that sweep s updates
// u[.][s & 1] and reads u[.][1 - (s & 1)] of its own rows above and below and of its own pair; only
// the pair's outer neighbour and the rows beyond the strip come from shared memory. Rows are
// stored there with even columns first, so that consecutive threads touch consecutive words.
#pragma once

// Measured on a B200, per V-cycle against the tile form as it then was: 57 -> 28 us at 255^2 and 28 -> 13 us
// at 63^2 (double). Per slice at 255^2, the coefficient kernel's 26 us (beside the Poisson solves outside a
// profile) included: 192 -> 148 us double, 158 -> 130 us mixed; at 63^2 with 7 V-cycles 213 -> 146 us.
//
// (included by mg.cuh, whose barrier polls it uses; levels and shared-memory plan: mgcl_plan.hpp)

namespace hpq {

constexpr long long kClWaits = 1 << 20;  // polls of an mbarrier (each suspends for up to microseconds)

// element (i, j) of a component plane in 0-based valid indices
template <class IO>
struct ClView {
    IO* p[2];
    int pitch;
    int off;
    __device__ IO* at(int c, int i, int j) const { return p[c] + (ptrdiff_t)(j + off) * pitch + (i + off); }
};

__device__ __forceinline__ void cl_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cl_bar_warps(int id, int nwarps) {
    asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(nwarps * 32) : "memory");
}
// shared::cluster address of a shared-memory element of block `rank`, and accesses through it
__device__ __forceinline__ uint32_t cl_map(const void* p, int rank) {
    uint32_t q;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(q) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return q;
}
__device__ __forceinline__ void cl_st(uint32_t a, double v) { asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }
__device__ __forceinline__ void cl_st(uint32_t a, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void cl_st(uint32_t a, int v) { asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void cl_ld(uint32_t a, double& v) { asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory"); }
__device__ __forceinline__ void cl_ld(uint32_t a, float& v) { asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory"); }

// store to another block's shared memory that counts its bytes on that block's mbarrier
__device__ __forceinline__ void cl_st_async(uint32_t a, double v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
                 "l"(__double_as_longlong(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void cl_st_async(uint32_t a, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a),
                 "r"(__float_as_int(v)), "r"(bar) : "memory");
}

// Shared words of one block beside the levels' planes
struct ClShared {
    unsigned long long bar[2][2];  // mbarriers of the rows from above [0] and below [1], used alternately
    unsigned long long copy;       // mbarrier of the coefficient copy
    unsigned long long norm;       // largest residual of the block (bits of a double)
    int go;    // 1: another V-cycle, 0: done, -1: a wait ran out; written by block 0 of the cluster
    int dead;  // a wait of this block ran out: no further waits
};
// Exchanges with the block above and below so far: the n-th uses mbarrier n & 1 in its phase n >> 1. A
// block sends for exchange n + 1 only after it has the neighbour's rows of exchange n, which the
// neighbour sends only after its own wait for exchange n - 1, so that the two mbarriers suffice.
struct ClSeq {
    int n[2];
};

extern __shared__ __align__(16) unsigned char cl_smem[];

template <class R, bool CELL>
struct ClSolve {
    const ClLev<R>* lev;  // shared memory
    ClShared* sh;
    int* err;
    int nl, rank, cs, ns_bottom, lm, nm;
    unsigned matrix;

    enum { LOAD = 0, ZERO = 1, INTERP = 2 };

    // barrier of the threads that work on level l: the block (DIST) or the level's warps
    template <bool DIST>
    __device__ __forceinline__ void sync_block(int l, int nwarps) const {
        if (DIST) __syncthreads(); else cl_bar_warps(1 + l, nwarps);
    }
    __device__ __forceinline__ void sync_cluster() const {
        if (cs > 1) cl_barrier(); else __syncthreads();
    }
    // Waits until the rows of an exchange have arrived (bounded; the phase alternates every second use)
    __device__ __forceinline__ void wait_rows(int dir, int n) const {
        const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&sh->bar[dir][n & 1]);
        const uint32_t parity = (n >> 1) & 1;
        uint32_t done = 0;
        for (long long it = 0;; ++it) {
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                         "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
            if (done || *(volatile int*)&sh->dead) return;
            if (it > kClWaits) {
                sh->dead = 1;
                atomicExch(err, 1);
                return;
            }
        }
    }
    // (bounded: a copy that does not arrive ends in the solve's error flag)
    __device__ __forceinline__ void wait_copy(uint32_t bar) const {
        uint32_t done = 0;
        for (long long it = 0; !done && it <= kClWaits; ++it)
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
                         "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar) : "memory");
        if (!done) {
            sh->dead = 1;
            atomicExch(err, 1);
        }
    }
    __device__ __forceinline__ void expect_rows(int dir, int n, uint32_t bytes) const {
        const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&sh->bar[dir][n & 1]);
        asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    }

    // a thread's place on a level: row group g, column pair k, first local and global row
    struct Place {
        int kp, rs, k, r0, grow;
        bool act;
    };
    template <int RT, bool DIST>
    __device__ __forceinline__ Place place(const ClLev<R>& L) const {
        Place t;
        t.kp = L.kp;
        t.rs = 2 * t.kp + 2;
        const int g = (int)((threadIdx.x * L.magic) >> 22);
        t.k = (int)threadIdx.x - g * t.kp;
        t.r0 = g * RT;
        t.grow = (DIST ? rank * L.rp : 0) + t.r0;
        t.act = g < L.ng;
        return t;
    }

    // Restriction to level l + 1 of a plane of level l in phi layout (row 0 at `src`; the residual,
    // zero on colour 1, or with ALL the coefficient). A thread makes the coarse points under its own
    // rows and column pair, so that the block's coarse rows come from its own fine rows and,
    // node-centred, the next block's first row (in xrow). `dst` is the coarse plane's first element,
    // rows of `drow` elements, odd columns from `dodd` on.
    template <int RT, bool DIST, bool ALL>
    __device__ __forceinline__ void restrict_plane(const ClLev<R>& L, const ClLev<R>& C, const Place& t, unsigned src,
                                                   unsigned dst, int drow, int dodd, unsigned xofs) const {
        R* sm = reinterpret_cast<R*>(cl_smem);
        const int cny = C.ny;
        if (!t.act || t.k >= C.nx) return;
        const bool remote = DIST && !C.dist && rank > 0;
        const int base = DIST && C.dist ? rank * (L.rp / 2) : 0;  // first coarse row of the plane at dst
        R* d = sm + dst + (t.k & 1) * dodd + (t.k >> 1) - base * drow;
        const uint32_t dr = remote ? cl_map(d, 0) : 0u;
        const R* xrow = sm + xofs;
        const int rp = L.rp;
        const int e0 = t.k, e1 = t.k + 1, o0 = t.kp + 2 + t.k;
        const R* a = sm + src + t.r0 * t.rs;
        const int q0 = t.grow & 1;
#pragma unroll
        for (int p = 0; p < (RT + 1) / 2; ++p) {
            const int q = RT > 1 ? 2 * p : 0;
            if (RT == 1 && q0) continue;
            const int cj = (t.grow + q) >> 1;
            if (cj >= cny) continue;
            const R *f = a + q * t.rs, *b = f + t.rs;
            R v;
            if (CELL) {
                v = ALL ? R(0.25) * (f[e0] + f[o0] + b[e0] + b[o0]) : R(0.25) * (f[e0] + b[o0]);
            } else {
                const R* c = (DIST && t.r0 + q + 2 == rp && cs > 1) ? xrow : b + t.rs;
                if (ALL)
                    v = R(1. / 16.) * (f[e0] + R(2.) * f[o0] + f[e1] + R(2.) * b[e0] + R(4.) * b[o0] + R(2.) * b[e1] +
                                       c[e0] + R(2.) * c[o0] + c[e1]);
                else
                    v = R(1. / 16.) * ((f[e0] + f[e1]) + (c[e0] + c[e1]) + R(4.) * b[o0]);
            }
            if (remote) cl_st(dr + (uint32_t)(cj * drow * (int)sizeof(R)), v);
            else d[cj * drow] = v;
        }
    }

    // Smoothing of level l: initial guess (in shared memory, zero, or that plus the interpolated
    // correction of level l + 1), nsw colour sweeps, and with `tail` the residual and its
    // restriction to the right-hand side of level l + 1. Returns the thread's largest |residual|.
    // Every thread of the block (DIST) or of the level's warps calls.
    template <int RT, bool DIST>
    __device__ __noinline__ double phase(int l, int init, int nsw, bool tail, ClSeq* seq) const {
        R* sm = reinterpret_cast<R*>(cl_smem);
        const ClLev<R>& L = lev[l];
        const Place t = place<RT, DIST>(L);
        const int nwarps = L.nwarps, lny = L.ny, lnx = L.nx, rp = L.rp;
        const int kp = t.kp, rs = t.rs, k = t.k;
        const int par = t.grow & 1;
        const R fx = L.facx, ratio = L.ratio;
        // words of the two columns of the pair: for rows q even [0], odd [1] holds colour 0's column
        // (colour 1's is the other), and of the outer neighbour on that column's side
        const int own0 = par ? kp + 2 + k : k, own1 = par ? k : kp + 2 + k;
        const int out0 = par ? k + 1 : kp + 1 + k, out1 = par ? kp + 1 + k : k + 1;
        const int rh0 = par ? kp + k : k, rh1 = par ? k : kp + k;
        R* phi = sm + L.phi + (t.r0 + 1) * rs;
        // neighbours of this block on the level, and this thread's share in the exchange with them
        const bool has_up = DIST && cl_joined(rank, cs, rp, lny, CELL);
        const bool has_dn = DIST && cl_joined(rank + 1, cs, rp, lny, CELL);
        const bool top = has_up && t.act && t.r0 == 0;
        const bool bot = has_dn && t.act && t.r0 + RT == rp;
        int nu = 0, nd = 0;
        if (DIST) { nu = seq->n[0]; nd = seq->n[1]; }
        // halo rows of the neighbours that mirror this block's first and last row, their mbarriers
        const uint32_t up_row = top ? cl_map(sm + L.phi + (rp + 1) * rs, rank - 1) : 0u;
        const uint32_t dn_row = bot ? cl_map(sm + L.phi, rank + 1) : 0u;
        const uint32_t up_bar = top ? cl_map(&sh->bar[1][0], rank - 1) : 0u;
        const uint32_t dn_bar = bot ? cl_map(&sh->bar[0][0], rank + 1) : 0u;
        const uint32_t row_bytes = (uint32_t)(kp * sizeof(R));
        // (the neighbour counts its exchanges with this block as this block does)
        auto send = [&](int q, int at, R v) {
            if (DIST && q == 0 && top) cl_st_async(up_row + at * (uint32_t)sizeof(R), v, up_bar + (nu & 1) * 8u);
            if (DIST && q == RT - 1 && bot) cl_st_async(dn_row + at * (uint32_t)sizeof(R), v, dn_bar + (nd & 1) * 8u);
        };
        // end of a step that sent one colour of the boundary rows
        auto exchange = [&]() {
            if (DIST) {
                if (threadIdx.x == 0) {
                    if (has_up) expect_rows(0, nu, row_bytes);
                    if (has_dn) expect_rows(1, nd, row_bytes);
                }
                __syncthreads();
                if (top) wait_rows(0, nu);
                if (bot) wait_rows(1, nd);
                nu += has_up;
                nd += has_dn;
            } else {
                cl_bar_warps(1 + l, nwarps);
            }
        };
        R u[RT][2], rv[RT][2], cx[RT][2];  // by colour: solution, rhs / diagonal, -facx / diagonal
        const R* rhs = sm + L.rhs + t.r0 * 2 * kp;
        const R* inv = sm + L.inv + t.r0 * 2 * kp;
        const R* low = sm + L.low + t.r0 * 2 * kp;
#pragma unroll
        for (int q = 0; q < RT; ++q) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int at = q * 2 * kp + (((q + e) & 1) ? rh1 : rh0);
                const R d = t.act ? inv[at] : R(0);
                rv[q][e] = t.act ? rhs[at] * d : R(0);
                cx[q][e] = -fx * d;
            }
            u[q][0] = R(0);
            u[q][1] = (t.act && init != ZERO) ? phi[q * rs + ((q & 1) ? own0 : own1)] : R(0);
        }
        auto store = [&](int q, int e) {
            const int at = ((q + e) & 1) ? own1 : own0;
            phi[q * rs + at] = u[q][e];
            send(q, at, u[q][e]);
        };
        if (init == INTERP) {
            const ClLev<R>& C = lev[l + 1];
            const int rsc = 2 * C.kp + 2;
            const int cphi = C.phi;
            const bool cdist = C.dist;
            if (DIST && !cdist && rank > 0) {
                // the rows that this block reads of the coarse solution of block 0, into the same place here
                const int c0 = rank * (rp / 2) - 1, c1 = min(c0 + rp / 2 + 2, C.ny + 1);  // rows c0 .. c1 - 1
                const int n = (c1 - c0) * rsc, o = cphi + (c0 + 1) * rsc;
                const uint32_t src = cl_map(sm + o, 0);
                for (int i = threadIdx.x; i < n; i += kClThreads) cl_ld(src + i * (uint32_t)sizeof(R), sm[o + i]);
                __syncthreads();
            }
            // colour 1 lies on even rows in odd columns (between two coarse rows) and on odd rows in even
            // columns (between two coarse columns)
            const int a1 = (k & 1) ? C.kp + 2 + (k >> 1) : (k >> 1);              // coarse column k
            const int a0 = (k & 1) ? ((k - 1) >> 1) : C.kp + 2 + ((k - 1) >> 1);  // coarse column k - 1
            const R* cb = sm + cphi + rsc;
            const int cbase = DIST && cdist ? rank * (rp / 2) : 0, crp = C.rp;
            if (t.act) {
#pragma unroll
                for (int q = 0; q < RT; ++q) {
                    const int row = t.grow + q;
                    const R* c1 = cb + cl_coarse_row(row, cbase, crp) * rsc;
                    R a;
                    if (CELL) a = c1[a1];
                    else a = (row & 1) ? (c1[a0] + c1[a1]) * R(0.5) : (c1[a1 - rsc] + c1[a1]) * R(0.5);
                    u[q][1] += cx[q][1] != R(0) ? a : R(0);  // (zero outside the grid)
                }
            }
        }
        if (init != ZERO) {
            if (t.act) {
#pragma unroll
                for (int q = 0; q < RT; ++q) store(q, 1);
            }
            exchange();
        }
        // (cell-centred: 4/3 of the inner neighbours in the first and last column and row)
        auto ex = [&](int q, int e) -> R {
            const int col = 2 * k + ((e ^ (par + q)) & 1);
            return (col == 0 || col == lnx - 1) ? R(4. / 3.) : R(1);
        };
        auto ey = [&](int q) -> R { return (t.grow + q == 0 || t.grow + q == lny - 1) ? R(4. / 3.) : R(1); };
        auto neighbours = [&](int q, int e, R& h, R& v) {
            const int own = ((q + e) & 1) ? own1 : own0, out = ((q + e) & 1) ? out1 : out0;
            h = u[q][1 - e] + phi[q * rs + out];
            R a, b;
            if (q > 0) a = u[q > 0 ? q - 1 : 0][1 - e]; else a = phi[-rs + own];
            if (q < RT - 1) b = u[q < RT - 1 ? q + 1 : q][1 - e]; else b = phi[RT * rs + own];
            v = a + b;
            if (CELL) { h *= ex(q, e); v *= ey(q); }
        };
        auto sweep = [&](auto colour, bool zero, bool first) {
            constexpr int e = decltype(colour)::value;
            if (t.act) {
                if (e == 0 && zero) {
#pragma unroll
                    for (int q = 0; q < RT; ++q) u[q][0] = rv[q][0];
                } else {
                    R n[RT];
#pragma unroll
                    for (int q = 0; q < RT; ++q) {
                        R h, v;
                        neighbours(q, e, h, v);
                        const R w = fma(ratio, v, h);
                        // (level 0 in single precision: the low part of the weight, once per phase, as it
                        // changes with the solution by rounding only)
                        if (std::is_same<R, float>::value && first && l == 0)
                            rv[q][e] = fma(low[q * 2 * kp + (((q + e) & 1) ? rh1 : rh0)], w, rv[q][e]);
                        n[q] = fma(cx[q][e], w, rv[q][e]);
                    }
#pragma unroll
                    for (int q = 0; q < RT; ++q) u[q][e] = n[q];
                }
#pragma unroll
                for (int q = 0; q < RT; ++q) store(q, e);
            }
            exchange();
        };
        for (int s = 0; s < nsw; s += 2) {
            sweep(std::integral_constant<int, 0>{}, s == 0 && init == ZERO, s == 0);
            sweep(std::integral_constant<int, 1>{}, false, s == 0);
        }
        R worst = 0;
        if (tail) {
            // residual of colour 0: the diagonal times the change that a further sweep would make (formed
            // with the sweeps' own arithmetic, it goes to zero in single precision too, where rhs + a phi -
            // Lap(phi) stalls at the rounding of the inverse diagonal). It takes the place of phi in shared
            // memory, whose colour 0 no neighbour reads any more, while the restriction reads it
            const ClLev<R>& C = lev[l + 1];
            if (t.act) {
                const R* dia = sm + L.dia + t.r0 * kp + k;
                const uint32_t xr = (!CELL && top) ? cl_map(sm + L.xrow, rank - 1) : 0u;
#pragma unroll
                for (int q = 0; q < RT; ++q) {
                    const int own = (q & 1) ? own1 : own0;
                    R h, v;
                    neighbours(q, 0, h, v);
                    const R r = dia[q * kp] * (fma(cx[q][0], fma(ratio, v, h), rv[q][0]) - u[q][0]);
                    worst = fmax(worst, fabs(r));
                    phi[q * rs + own] = r;
                    if (DIST && !CELL && q == 0 && top) cl_st_async(xr + own * (uint32_t)sizeof(R), r, up_bar + (nu & 1) * 8u);
                    // (the row below is not needed there, but every exchange goes both ways: a block that had
                    // nothing to wait for could get two exchanges ahead and count into an mbarrier whose
                    // phase has not ended; colour 0 of the halo row is free here)
                    if (DIST && !CELL && q == RT - 1 && bot) cl_st_async(dn_row + own * (uint32_t)sizeof(R), r, dn_bar + (nd & 1) * 8u);
                }
            }
            if (DIST && !CELL && cs > 1) {
                if (threadIdx.x == 0) {
                    if (has_up) expect_rows(0, nu, row_bytes);
                    if (has_dn) expect_rows(1, nd, row_bytes);
                }
                __syncthreads();
                if (top) wait_rows(0, nu);
                // (and the threads whose coarse row reaches into xrow)
                if (has_dn && t.act && t.r0 + RT >= rp - (RT == 1 ? 1 : 0)) wait_rows(1, nd);
                nu += has_up;
                nd += has_dn;
            } else {
                sync_block<DIST>(l, nwarps);
            }
            restrict_plane<RT, DIST, false>(L, C, t, L.phi + rs, C.rhs, 2 * C.kp, C.kp, L.xrow);
            // the right-hand side of a level of block 0 comes from the whole cluster
            if (DIST && !C.dist) sync_cluster(); else sync_block<DIST>(l, nwarps);
            if (l == 0 && t.act) {
#pragma unroll
                for (int q = 0; q < RT; ++q) phi[q * rs + ((q & 1) ? own1 : own0)] = u[q][0];
            }
        }
        if (DIST) {
            seq->n[0] = nu;
            seq->n[1] = nd;
            // the rows awaited by the boundary threads are there for all threads, and no thread sends for the
            // next exchange before (the next level's boundary threads are others)
            if (!tail) __syncthreads();
        }
        return (double)worst;
    }

    // Set-up of level l, whose coefficient is in place: inverse diagonals, and the coefficient of
    // level l + 1 (average_down_acoef, HpMultiGrid.cpp:1640-1700)
    template <int RT, bool DIST>
    __device__ __noinline__ void coefficient(int l) const {
        R* sm = reinterpret_cast<R*>(cl_smem);
        const ClLev<R>& L = lev[l];
        const Place t = place<RT, DIST>(L);
        const R* acf = sm + L.cacf + t.r0 * t.rs;
        if (t.act) {
            const uint32_t xr = (DIST && t.r0 == 0 && rank > 0) ? cl_map(sm + L.cxrow, rank - 1) : 0u;
#pragma unroll
            for (int q = 0; q < RT; ++q)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int i = 2 * t.k + c, j = t.grow + q, at = c ? t.kp + 2 + t.k : t.k;
                    const R a = acf[q * t.rs + at];
                    R c0 = -(a + R(2.) * (L.facx + L.facy));
                    if (CELL && (i == 0 || i == L.nx - 1)) c0 -= R(2.) * L.facx;
                    if (CELL && (j == 0 || j == L.ny - 1)) c0 -= R(2.) * L.facy;
                    sm[L.cinv + ((t.r0 + q) * 2 + c) * t.kp + t.k] = (i < L.nx && j < L.ny) ? R(1.) / c0 : R(0);
                    if (DIST && q == 0 && xr) cl_st(xr + at * (uint32_t)sizeof(R), a);
                }
        }
        if (l + 1 == nl) return;
        if (DIST) sync_cluster(); else sync_block<false>(l, L.nwarps);
        const ClLev<R>& C = lev[l + 1];
        restrict_plane<RT, DIST, true>(L, C, t, L.cacf, C.cacf, 2 * C.kp + 2, C.kp + 2, L.cxrow);
        if (DIST) sync_cluster(); else sync_block<false>(l, L.nwarps);
    }

    template <bool DIST>
    __device__ double run_phase(int l, int init, int nsw, bool tail, ClSeq* seq = nullptr) const {
        switch (lev[l].rt) {
            case 1: return phase<1, DIST>(l, init, nsw, tail, seq);
            case 2: return phase<2, DIST>(l, init, nsw, tail, seq);
            case 4: return phase<4, DIST>(l, init, nsw, tail, seq);
            default: return phase<8, DIST>(l, init, nsw, tail, seq);
        }
    }
    template <bool DIST>
    __device__ void run_coefficient(int l) const {
        switch (lev[l].rt) {
            case 1: return coefficient<1, DIST>(l);
            case 2: return coefficient<2, DIST>(l);
            case 4: return coefficient<4, DIST>(l);
            default: return coefficient<8, DIST>(l);
        }
    }

    // The matrix of levels lm .. nl - 1 applied by `nthreads` threads: correction of level lm from its
    // right-hand side (both in storage order of the right-hand side)
    __device__ __forceinline__ void apply_matrix(int nthreads) const {
        R* sm = reinterpret_cast<R*>(cl_smem);
        const ClLev<R>& L = lev[lm];
        const int parts = nthreads >= 8 * nm ? 8 : nthreads >= 4 * nm ? 4 : nthreads >= 2 * nm ? 2 : 1;
        const R* f = sm + L.rhs;
        const int kp = L.kp, p = threadIdx.x & (parts - 1);
        const int step = nthreads / parts, rounds = (nm + step - 1) / step;
        for (int q = 0; q < rounds; ++q) {
            const int i = (int)threadIdx.x / parts + q * step;
            const R* m = sm + matrix + (i < nm ? i : 0) * nm;
            R a = 0, b = 0;
            int j = p;
            for (; j + parts < nm; j += 2 * parts) {
                a = fma(m[j], f[j], a);
                b = fma(m[j + parts], f[j + parts], b);
            }
            if (j < nm) a = fma(m[j], f[j], a);
            a += b;
            for (int d = 1; d < parts; d <<= 1) a += __shfl_xor_sync(0xffffffffu, a, d);
            if (p == 0 && i < nm) {
                const int r2 = i / kp, k = i - r2 * kp;  // (row, column parity)
                sm[L.phi + ((r2 >> 1) + 1) * (2 * kp + 2) + ((r2 & 1) ? kp + 2 + k : k)] = a;
            }
        }
    }

    // levels [l0, nl) in block 0: a level is run by its own warps; a warp without work on level l
    // waits for it at the barrier that opens the up-sweep of level l - 1
    __device__ void bottom(int l0) const {
        const int warp = threadIdx.x >> 5, last = nl - 1;
        if (lm == l0) { apply_matrix(kClThreads); return; }
        if (warp >= lev[l0].nwarps) return;
        int l = l0;
        for (; l < last && l < lm && warp < lev[l].nwarps; ++l) run_phase<false>(l, ZERO, 4, true);
        if (l == lm) apply_matrix(lev[l - 1].nwarps * 32);
        else if (l == last && warp < lev[l].nwarps) run_phase<false>(last, ZERO, ns_bottom, false);
        for (int m = l - 1; m >= l0; --m) {
            cl_bar_warps(1 + m, lev[m].nwarps);
            run_phase<false>(m, INTERP, 4, false);
        }
    }
    // Column j of the matrix, by one warp: the V-cycle of levels lm .. nl - 1 (4 sweeps, residual and
    // restriction down, ns_bottom sweeps on the coarsest level, interpolation and 4 sweeps up) on
    // the unit right-hand side j. `w`: scratch of the warp, kClWarpScratch elements.
    __device__ void matrix_column(int j, R* w, R* out) const {
        R* sm = reinterpret_cast<R*>(cl_smem);
        const int lane = threadIdx.x & 31;
        // per level: rhs (storage order), phi with a border of zeros, (nx + 2) x (ny + 2)
        int ofs[6], n = nl - lm, o = 0;
        for (int q = 0; q < n; ++q) {
            const ClLev<R>& L = lev[lm + q];
            ofs[q] = o;
            o += L.rp * 2 * L.kp + (L.nx + 2) * (L.ny + 2);
        }
        for (int i = lane; i < o; i += 32) w[i] = R(0);
        __syncwarp();
        if (lane == 0) w[j] = R(1);
        __syncwarp();
        auto frhs = [&](int q) { return w + ofs[q]; };
        auto fphi = [&](int q) { return w + ofs[q] + lev[lm + q].rp * 2 * lev[lm + q].kp; };
        // a lane holds one point of a level (at most 32 points); the 5-point neighbours times their factors
        auto sides = [&](const ClLev<R>& L, const R* c, int x, int y) -> R {
            const int W = L.nx + 2;
            R h = c[-1] + c[1], v = c[-W] + c[W];
            if (CELL && (x == 0 || x == L.nx - 1)) h *= R(4. / 3.);
            if (CELL && (y == 0 || y == L.ny - 1)) v *= R(4. / 3.);
            return L.facx * h + L.facy * v;
        };
        auto at = [&](const ClLev<R>& L, int x, int y) { return (y * 2 + (x & 1)) * L.kp + (x >> 1); };
        auto sweeps = [&](int q, int ns) {
            const ClLev<R>& L = lev[lm + q];
            const int y = lane / L.nx, x = lane - y * L.nx;
            const bool in = y < L.ny;
            R* c = fphi(q) + (in ? (y + 1) * (L.nx + 2) + x + 1 : 0);
            const R f = in ? frhs(q)[at(L, x, y)] : R(0), d = in ? sm[L.cinv + at(L, x, y)] : R(0);
            for (int s = 0; s < ns; ++s) {
                if (in && ((x + y + s) & 1) == 0) *c = (f - sides(L, c, x, y)) * d;
                __syncwarp();
            }
        };
        for (int q = 0; q + 1 < n; ++q) {
            sweeps(q, 4);
            const ClLev<R>& L = lev[lm + q];
            const ClLev<R>& C = lev[lm + q + 1];
            auto residual = [&](int x, int y) -> R {  // of a point of colour 0
                const R* c = fphi(q) + (y + 1) * (L.nx + 2) + x + 1;
                R lap = R(-2.) * (L.facx + L.facy) * *c + sides(L, c, x, y);
                if (CELL && (x == 0 || x == L.nx - 1)) lap -= R(2.) * L.facx * *c;
                if (CELL && (y == 0 || y == L.ny - 1)) lap -= R(2.) * L.facy * *c;
                const R a = sm[L.cacf + y * (2 * L.kp + 2) + ((x & 1) ? L.kp + 2 : 0) + (x >> 1)];
                return frhs(q)[at(L, x, y)] + a * *c - lap;
            };
            const int y = lane / C.nx, x = lane - y * C.nx;
            if (y < C.ny) {
                R v;
                if (CELL) v = R(0.25) * (residual(2 * x, 2 * y) + residual(2 * x + 1, 2 * y + 1));
                else
                    v = R(1. / 16.) * (residual(2 * x, 2 * y) + residual(2 * x + 2, 2 * y) + residual(2 * x, 2 * y + 2) +
                                       residual(2 * x + 2, 2 * y + 2) + R(4.) * residual(2 * x + 1, 2 * y + 1));
                frhs(q + 1)[at(C, x, y)] = v;
            }
            __syncwarp();
        }
        sweeps(n - 1, ns_bottom);
        for (int q = n - 2; q >= 0; --q) {
            const ClLev<R>& L = lev[lm + q];
            const ClLev<R>& C = lev[lm + q + 1];
            const R* c = fphi(q + 1);
            auto cv = [&](int x, int y) { return c[(y + 1) * (C.nx + 2) + x + 1]; };
            const int y = lane / L.nx, x = lane - y * L.nx;
            if (y < L.ny && ((x + y) & 1)) {  // (the first sweep replaces colour 0)
                R v;
                if (CELL) v = cv(x >> 1, y >> 1);
                else v = (y & 1) ? (cv((x >> 1) - 1, y >> 1) + cv(x >> 1, y >> 1)) * R(0.5)
                                 : (cv(x >> 1, (y >> 1) - 1) + cv(x >> 1, y >> 1)) * R(0.5);
                fphi(q)[(y + 1) * (L.nx + 2) + x + 1] += v;
            }
            __syncwarp();
            sweeps(q, 4);
        }
        const ClLev<R>& L = lev[lm];
        const int y = lane / L.nx, x = lane - y * L.nx;
        if (y < L.ny) out[at(L, x, y) * nm + j] = fphi(0)[(y + 1) * (L.nx + 2) + x + 1];
        __syncwarp();
    }
    __device__ void bottom_coefficients(int l0) const {
        const int warp = threadIdx.x >> 5;
        for (int l = l0; l < nl && warp < lev[l].nwarps; ++l) run_coefficient<false>(l);
    }

    // level 0 from the slice arrays; returns the thread's largest |rhs|
    template <int RT, class V>
    __device__ __noinline__ double load(const V& sol, const V& rhs, int comp) const {
        R* sm = reinterpret_cast<R*>(cl_smem);
        const ClLev<R>& L = lev[0];
        const Place t = place<RT, true>(L);
        R w = 0;
        if (!t.act) return 0.0;
        R v[2][RT][2];
#pragma unroll
        for (int q = 0; q < RT; ++q)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int i = 2 * t.k + c, j = t.grow + q;
                const bool in = i < L.nx && j < L.ny;
                v[0][q][c] = in ? (R)*sol.at(comp, i, j) : R(0);
                v[1][q][c] = in ? (R)*rhs.at(comp, i, j) : R(0);
            }
#pragma unroll
        for (int q = 0; q < RT; ++q)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int at = c ? t.kp + 2 + t.k : t.k, r = t.r0 + q;
                sm[L.phi + (r + 1) * t.rs + at] = v[0][q][c];
                sm[L.rhs + (r * 2 + c) * t.kp + t.k] = v[1][q][c];
                w = fmax(w, fabs(v[1][q][c]));
            }
        return (double)w;
    }
    // coefficient of level 0 from the slice arrays (k_mg_cluster_coef)
    template <int RT, class V>
    __device__ void load_acf(const V& a0) const {
        R* sm = reinterpret_cast<R*>(cl_smem);
        const ClLev<R>& L = lev[0];
        const Place t = place<RT, true>(L);
        if (!t.act) return;
#pragma unroll
        for (int q = 0; q < RT; ++q)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int i = 2 * t.k + c, j = t.grow + q;
                if (i < L.nx && j < L.ny) sm[L.cacf + (t.r0 + q) * t.rs + (c ? t.kp + 2 + t.k : t.k)] = (R)*a0.at(0, i, j);
            }
    }
    template <int RT, class V>
    __device__ void save(const V& sol, int comp) const {
        R* sm = reinterpret_cast<R*>(cl_smem);
        const ClLev<R>& L = lev[0];
        const Place t = place<RT, true>(L);
        if (!t.act) return;
#pragma unroll
        for (int q = 0; q < RT; ++q)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int i = 2 * t.k + c, j = t.grow + q;
                if (i < L.nx && j < L.ny)
                    *sol.at(comp, i, j) = sm[L.phi + (t.r0 + q + 1) * t.rs + (c ? t.kp + 2 + t.k : t.k)];
            }
    }
};

template <class R>
__device__ __forceinline__ void cl_levels_to_shared(const ClArgs<R>& P, ClLev<R>* slev) {
    static_assert(sizeof(ClLev<R>) % 4 == 0, "copied by words");
    const int* src = reinterpret_cast<const int*>(P.lev);
    int* dst = reinterpret_cast<int*>(slev);
    for (int t = threadIdx.x; t < (int)(sizeof(ClLev<R>) / 4) * P.nl; t += kClThreads) dst[t] = src[t];
}

// Coefficient hierarchy of a solve, one cluster: restricts the coefficient, inverts the diagonals,
// forms the matrix of the smallest levels and writes each block's region (ClArgs::coef). It needs
// the slice's chi only, so the slice loop runs it beside the Poisson solves; in the solve it took
// 26 000 of 90 000 cycles at 255^2 in double.
template <class IO, class R, bool CELL>
__global__ void __launch_bounds__(kClThreads, 1) k_mg_cluster_coef(const __grid_constant__ ClArgs<R> P, ClView<IO> a0) {
    HPQ_PDL_ENTRY();
    __shared__ ClLev<R> slev[kClMaxLevels];
    const int cs = P.cs, rank = (int)blockIdx.x;
    R* sm = reinterpret_cast<R*>(cl_smem);
    using S = ClSolve<R, CELL>;
    cl_levels_to_shared(P, slev);
    int4* z = reinterpret_cast<int4*>(cl_smem);
    for (unsigned t = threadIdx.x; t < P.celems * sizeof(R) / 16; t += kClThreads) z[t] = make_int4(0, 0, 0, 0);
    if (rank == 0 && threadIdx.x < 6 * kClMaxBlocks) P.slot[threadIdx.x] = ClNorm{};
    __syncthreads();
    const S s{slev, nullptr, nullptr, P.nl, rank, cs, P.ns_bottom, P.lm, P.nm, P.matrix};
    int nd = 0;
    while (nd < P.nl && slev[nd].dist) ++nd;
    switch (slev[0].rt) {
        case 1: s.template load_acf<1>(a0); break;
        case 2: s.template load_acf<2>(a0); break;
        case 4: s.template load_acf<4>(a0); break;
        default: s.template load_acf<8>(a0); break;
    }
    s.sync_cluster();  // every block has started: its shared memory may be written
    for (int l = 0; l < nd; ++l) s.template run_coefficient<true>(l);
    if (rank == 0) {
        if (nd < P.nl) s.bottom_coefficients(nd);
        __syncthreads();
        if (P.lm < P.nl) {
            const int warp = threadIdx.x >> 5;
            R* w = sm + P.celems - (kClThreads / 32 - warp) * kClWarpScratch;
            const ClLev<R>& L = slev[P.lm];
            for (int i = threadIdx.x; i < P.nm * P.nm; i += kClThreads) P.coef[P.matrix + i] = R(0);
            __syncthreads();
            for (int j = warp; j < P.nm; j += kClThreads / 32) {
                const int r2 = j / L.kp, x = 2 * (j - r2 * L.kp) + (r2 & 1);
                if (x < L.nx && (r2 >> 1) < L.ny) s.matrix_column(j, w, P.coef + P.matrix);
            }
        }
    }
    __syncthreads();  // (the last level's diagonals, where it is split, are behind no other barrier)
    R* out = P.coef + (size_t)rank * P.coef_elems;
    for (int l = 0; l < (rank == 0 ? min(P.nl, P.lm) : nd); ++l) {
        const ClLev<R>& L = slev[l];
        for (int i = threadIdx.x; i < L.rp * 2 * L.kp; i += kClThreads) out[L.inv + i] = sm[L.cinv + i];
        const int row0 = L.dist ? rank * L.rp : 0;
        if (l == 0 && std::is_same<R, float>::value) {
            for (int i = threadIdx.x; i < L.rp * 2 * L.kp; i += kClThreads) {
                const int r2 = i / L.kp, k = i - r2 * L.kp, c = r2 & 1, x = 2 * k + c, y = row0 + (r2 >> 1);
                const R a = sm[L.cacf + (r2 >> 1) * (2 * L.kp + 2) + (c ? L.kp + 2 + k : k)];
                out[L.low + i] = mg_weight_low<R>(CELL && (x == 0 || x == L.nx - 1), CELL && (y == 0 || y == L.ny - 1),
                                                  a, L.facx, L.ratio, -L.facx * sm[L.cinv + i]);
            }
        }
        for (int i = threadIdx.x; i < L.rp * L.kp; i += kClThreads) {
            const int r = i / L.kp, k = i - r * L.kp, c = (row0 + r) & 1, x = 2 * k + c, y = row0 + r;
            R d = -(sm[L.cacf + r * (2 * L.kp + 2) + (c ? L.kp + 2 + k : k)] + R(2.) * (L.facx + L.facy));
            if (CELL && (x == 0 || x == L.nx - 1)) d -= R(2.) * L.facx;
            if (CELL && (y == 0 || y == L.ny - 1)) d -= R(2.) * L.facy;
            out[L.dia + i] = x < L.nx && y < L.ny ? d : R(0);
        }
    }
    s.sync_cluster();  // no block leaves while another may still reach its shared memory
}

// gridDim.x = 2 clusters of P.cs blocks; cluster c solves component c. IO: type of the slice arrays,
// R: type of the solve (double for FP64 accuracy in a single-precision slice loop).
template <class IO, class R, bool CELL>
__global__ void __launch_bounds__(kClThreads, 1)
    k_mg_cluster(const __grid_constant__ ClArgs<R> P, ClView<IO> sol, ClView<IO> rhs) {
    HPQ_PDL_ENTRY();
    __shared__ ClLev<R> slev[kClMaxLevels];
    __shared__ ClShared sh;
    const int cs = P.cs, rank = (int)blockIdx.x % cs, comp = (int)blockIdx.x / cs;
    using S = ClSolve<R, CELL>;
    const unsigned copied = (rank == 0 ? P.coef_elems : P.dist_elems) * (unsigned)sizeof(R);
    const uint32_t copy_bar = (uint32_t)__cvta_generic_to_shared(&sh.copy);
    if (threadIdx.x == 0) {
        sh.go = 1;
        sh.dead = 0;
        sh.norm = 0;
        for (int d = 0; d < 4; ++d)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(&sh.bar[d >> 1][d & 1])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(copy_bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // this block's coefficients (the region of its shared memory from element 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(copy_bar), "r"(copied) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(cl_smem)),
                     "l"(P.coef + (size_t)rank * P.coef_elems), "r"(copied), "r"(copy_bar) : "memory");
    }
    cl_levels_to_shared(P, slev);
    {
        int4* z = reinterpret_cast<int4*>(cl_smem);
        for (unsigned t = P.coef_elems * sizeof(R) / 16 + threadIdx.x; t < P.elems * sizeof(R) / 16; t += kClThreads)
            z[t] = make_int4(0, 0, 0, 0);
    }
    __syncthreads();
    const S s{slev, &sh, &P.ctl->mgp_bar_err, P.nl, rank, cs, P.ns_bottom, P.lm, P.nm, P.matrix};
    int nd = 0;  // levels split over the cluster (at least level 0)
    while (nd < P.nl && slev[nd].dist) ++nd;
    auto sync_all = [&]() { if (cs > 1) cl_barrier(); else __syncthreads(); };
    double rmax;
    switch (slev[0].rt) {
        case 1: rmax = s.template load<1>(sol, rhs, comp); break;
        case 2: rmax = s.template load<2>(sol, rhs, comp); break;
        case 4: rmax = s.template load<4>(sol, rhs, comp); break;
        default: rmax = s.template load<8>(sol, rhs, comp); break;
    }
    s.wait_copy(copy_bar);
    sync_all();  // every block has started: its shared memory may be written
    // largest |residual| of the block -> global; the decision is taken by block 0 of each cluster once
    // every block's value of the iteration is there
    auto block_max = [&](double v) {  // valid in thread 0
        const unsigned long long b = (unsigned long long)__double_as_longlong(v);
        const unsigned hi = (unsigned)(b >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)b : 0u);
        if ((threadIdx.x & 31) == 0) atomicMax(&sh.norm, ((unsigned long long)mh << 32) | ml);
        __syncthreads();
        double m = 0;
        if (threadIdx.x == 0) {
            m = __longlong_as_double((long long)sh.norm);
            sh.norm = 0;  // (the next use lies behind another barrier)
        }
        return m;
    };
    const int me = comp * kClMaxBlocks + rank;
    auto publish = [&](double worst, ClNorm* slot, int it) {
        const double m = block_max(worst);
        if (threadIdx.x == 0) {
            const ClNorm n = cl_norm((unsigned long long)__double_as_longlong(m), (unsigned)it + 1u);
            asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(slot + me), "l"(n.w[0]), "l"(n.w[1]) : "memory");
        }
    };
    auto slots = [&](int it) { return P.slot + (it & 1) * 2 * kClMaxBlocks; };
    ClNorm* const rhs_slots = P.slot + 4 * kClMaxBlocks;
    double target = 0, maxnorm = 0;  // warp 0 of block 0 of each cluster
    auto decide = [&](int it) {      // warp 0 of block 0 of each cluster
        const int lane = threadIdx.x & 31;
        int ok = 1;
        const int late = *(const volatile int*)&P.ctl->mgp_bar_err;  // (a wait of any block ran out)
        auto fetch = [&](const ClNorm* p, int iteration) -> double {
            ClNorm v{};
            if ((lane & 15) < cs) {
                for (long long n = 0;; ++n) {
                    asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.w[0]), "=l"(v.w[1]) : "l"(p + lane) : "memory");
                    if (cl_norm_arrived(v, (unsigned)iteration + 1u)) break;
                    if ((n & 1023) == 1023 && *(const volatile int*)&P.ctl->mgp_bar_err) { ok = 0; break; }
                    if (n > kBarrierSpins) { atomicExch(&P.ctl->mgp_bar_err, 1); ok = 0; break; }
                }
            }
            __syncwarp();
            const unsigned hi = cl_norm_hi(v), mh = __reduce_max_sync(0xffffffffu, hi);
            const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? cl_norm_lo(v) : 0u);
            return __longlong_as_double((long long)(((unsigned long long)mh << 32) | ml));
        };
        const double w = fetch(slots(it), it);
        if (it == 0) {
            const double m = fetch(rhs_slots, 0);
            maxnorm = m >= w ? m : w;
            target = fmax(P.tol_abs, fmax(P.tol_rel, 1.e-16) * maxnorm);
        }
        ok = __all_sync(0xffffffffu, ok && !late);
        int go = 1, status = 0;
        if (it == 0) go = !(w <= target);
        else if (w <= target) go = 0;
        else if (w > 1.e20 * maxnorm) { go = 0; status = 2; }
        else if (it >= P.maxiter) { go = 0; status = 1; }
        if (!ok) go = -1;
        if (lane < cs) cl_st(cl_map(&sh.go, lane), go);
        if (comp == 0 && lane == 0) {
            Ctl* ctl = P.ctl;
            if (it == 0) { ctl->mg_target = target; ctl->mg_maxnorm = maxnorm; }
            else ctl->mg_total_iters += 1;
            ctl->mg_iter = it;
            ctl->mg_go = 0;
            if (status && !ctl->mg_status) ctl->mg_status = status;
        }
    };
    const int last = P.nl - 1;
    // first smoothing, then V-cycles: the up-sweep of level 0 and the next down-sweep are 8
    // consecutive sweeps. The norm of a V-cycle travels between the clusters while the next one
    // descends; a descent after the last V-cycle is thrown away.
    ClSeq seq{{0, 0}};
    publish(rmax, rhs_slots, 0);
    publish(s.template run_phase<true>(0, S::LOAD, 4, true, &seq), slots(0), 0);
    for (int it = 0;;) {
        if (nd == 1) {
            if (rank == 0 && threadIdx.x < 32) decide(it);
            sync_all();
        }
        for (int l = 1; l < nd; ++l) {
            if (l == last) s.template run_phase<true>(l, S::ZERO, P.ns_bottom, false, &seq);
            else s.template run_phase<true>(l, S::ZERO, 4, true, &seq);
            // taken once the norms have had level 1's time to arrive, known to the cluster by the barrier
            // that ends the last split level's descent
            if (l == 1) {
                if (rank == 0 && threadIdx.x < 32) decide(it);
                if (nd == 2 || nd == P.nl) sync_all();
            }
        }
        if (sh.go != 1) break;
        if (nd < P.nl) {
            if (rank == 0) s.bottom(nd);
            sync_all();
        }
        for (int l = (nd == P.nl ? nd - 2 : nd - 1); l >= 1; --l) s.template run_phase<true>(l, S::INTERP, 4, false, &seq);
        const double worst = s.template run_phase<true>(0, S::INTERP, 8, true, &seq);
        ++it;
        publish(worst, slots(it), it);
    }
    if (sh.go == 0) {
        __syncthreads();
        switch (slev[0].rt) {
            case 1: s.template save<1>(sol, comp); break;
            case 2: s.template save<2>(sol, comp); break;
            case 4: s.template save<4>(sol, comp); break;
            default: s.template save<8>(sol, comp); break;
        }
    }
    sync_all();  // no block leaves while another may still reach its shared memory
}

}  // namespace hpq

// Host side of the cluster-resident multigrid (mgcl.cuh): the levels of a grid, which grids take the
// cluster form, and its shared-memory plan. Plain C++, so that the plans of all grids can be checked
// without a GPU.
#pragma once

#include <algorithm>
#include <cstddef>
#include <map>
#include <mutex>
#include <set>
#include <type_traits>
#include <vector>

namespace hpq {

struct Ctl;

struct MGLev {
    int w, h;               // full box (cell: n; node: N+2)
    int vlo, vhi_i, vhi_j;  // valid box [vlo, vhi]
};

// Levels of an nx x ny grid: cell-centred (nx even) or node-centred, halved while both sides allow it
inline std::vector<MGLev> mg_levels(int nx, int ny) {
    const bool cell = nx % 2 == 0;
    std::vector<MGLev> lev;
    int lx, ly;
    if (cell) { lx = nx - 1; ly = ny - 1; } else { lx = nx + 1; ly = ny + 1; }
    for (int l = 0; l < 40; ++l) {
        MGLev L;
        L.w = lx + 1; L.h = ly + 1;
        if (cell) { L.vlo = 0; L.vhi_i = lx; L.vhi_j = ly; }
        else { L.vlo = 1; L.vhi_i = lx - 1; L.vhi_j = ly - 1; }
        lev.push_back(L);
        const int len_x = lx + 1, len_y = ly + 1, minw = cell ? 2 : 4;
        if (len_x < 2 * minw || len_y < 2 * minw) break;
        if (cell) { if (len_x % 2 || len_y % 2) break; lx = len_x / 2 - 1; ly = len_y / 2 - 1; }
        else { if (lx % 2 || ly % 2) break; lx /= 2; ly /= 2; }
    }
    return lev;
}
// the bottom solve of HpMultiGrid's CPU build (HpMultiGrid.cpp:1584-1592): 16 sweeps, or the longest
// side of the coarsest level rounded up to an even count when that is more (grids that stop
// coarsening early, e.g. 100 x 72 -> 25 x 18)
inline int mg_bottom_sweeps(const std::vector<MGLev>& lev) {
    return std::max(16, (std::max(lev.back().w, lev.back().h) + 1) / 2 * 2);
}

constexpr int kClThreads = 512;
constexpr int kClMaxLevels = 12;
constexpr int kClMaxBlocks = 16;  // per cluster
constexpr int kClWarpScratch = 384;  // elements of matrix_column (levels of at most 32 storage places)

// Host and device code of this file
#ifdef __CUDACC__
#define HPQ_HD __host__ __device__
#else
#define HPQ_HD
#endif

// A norm that a block publishes for the others: the upper and the lower 32 bits of the double, each in a
// 64-bit word with the iteration number + 1, so that value and arrival are in the same word and the two
// words may be seen in any order
struct alignas(16) ClNorm {
    unsigned long long w[2];
};
HPQ_HD inline ClNorm cl_norm(unsigned long long bits, unsigned tag) {
    return {{(bits & ~0xffffffffull) | tag, (bits << 32) | tag}};
}
HPQ_HD inline bool cl_norm_arrived(const ClNorm& n, unsigned tag) { return (unsigned)n.w[0] == tag && (unsigned)n.w[1] == tag; }
HPQ_HD inline unsigned cl_norm_hi(const ClNorm& n) { return (unsigned)(n.w[0] >> 32); }
HPQ_HD inline unsigned cl_norm_lo(const ClNorm& n) { return (unsigned)(n.w[1] >> 32); }

// One level of the cluster form. Shared-memory planes (element offsets): a row of phi and xrow has
// 2 kp + 2 elements: even columns at [k], a zero, a zero, odd columns at [kp + 2 + k] (the zeros are
// the values outside the grid); phi has rp + 2 rows (halo rows above and below). rhs and inverse
// diagonal have rp rows of 2 kp elements (even columns, odd columns), the diagonal rp rows of the kp
// colour-0 points, where the residual is formed. Rows and columns beyond the grid hold zeros, also
// as inverse diagonal, so that the sweeps leave them at zero without a test. low (level 0 in single
// precision, laid out like inv): what rounding took from the weight facx / diagonal (mg_weight_low).
template <class R>
struct ClLev {
    int nx, ny;     // valid points
    int kp;         // column pairs
    unsigned magic; // ceil(2^22 / kp): threadIdx / kp by multiplication
    int rp;         // rows per block (all rows, rounded up to rt, on levels that run in block 0)
    int dist;       // rows split over the cluster
    int rt, ng;     // rows per thread, row groups per block: rt * ng = rp
    int nwarps;     // warps with work (levels of block 0)
    unsigned phi, rhs, inv, dia, low, xrow;
    unsigned cacf, cinv, cxrow;  // planes of k_mg_cluster_coef: full coefficient (phi layout), inverse diagonal
    R facx, facy, ratio;         // ratio = facy / facx
};

template <class R>
struct ClArgs {
    int nl, cs, ns_bottom, maxiter;
    int lm, nm;  // levels lm .. nl - 1 as one matrix of nm x nm (lm = nl: none)
    ClLev<R> lev[kClMaxLevels];
    Ctl* ctl;
    double tol_rel, tol_abs;
    ClNorm* slot;  // [3][2 * kClMaxBlocks]: norm of every block by iteration parity, then |rhs| (cleared per solve)
    // coefficient region of every block, in the order of its shared memory (from element 0): inverse
    // diagonals and coefficients of the split levels (dist_elems), in block 0 also those of its
    // own levels, then the matrix (coef_elems)
    R* coef;
    unsigned dist_elems, coef_elems, matrix;
    unsigned elems, celems;    // shared-memory elements in use (solve, k_mg_cluster_coef)
};

// Whether block `rank` exchanges rows of a level split into `rp` rows per block with the block above it. A
// node-centred level counts one row beyond its last: the finer level has 2 n + 1 rows over n, and a block
// with the last of them alone interpolates it from the row above, which lies in the block above.
HPQ_HD inline bool cl_joined(int rank, int cs, int rp, int ny, bool cell) { return rank > 0 && rank < cs && rank * rp < ny + (cell ? 0 : 1); }

// Row of a block's coarse plane (rows -1 .. crp) that interpolation reads for fine row `row`; base: the
// plane's first row. A thread may own rows beyond the grid, for which the plane of a level in block 0
// has none: it reads the last row's (and discards the value).
HPQ_HD inline int cl_coarse_row(int row, int base, int crp) {
    const int c = (row >> 1) - base;
    return c < crp ? c : crp;
}

// Solvers of this process, by device, whose two clusters are launched without a guarantee that both become
// resident. Each cluster waits for the other's norms, so such solvers could stop one another only if single
// halves held every place: with fewer solvers than places at least one place is left for a partner.
// A solver that would be one too many launches cooperatively (mg.cuh). (Not all do: ncu cannot
// profile a cooperative launch with clusters.)
class ClSeat {
public:
    ClSeat() = default;
    ClSeat(const ClSeat&) = delete;
    ClSeat& operator=(const ClSeat&) = delete;
    ~ClSeat() { give(); }
    // false: no seat, launch cooperatively. places: clusters of this solver that an idle GPU holds
    bool take(int device, int places) {
        give();
        std::lock_guard<std::mutex> lock(mutex());
        std::multiset<int>& taken = seats()[device];
        const int fewest = taken.empty() ? places : std::min(places, *taken.begin());
        if ((int)taken.size() + 1 >= fewest) return false;
        taken.insert(places);
        device_ = device;
        places_ = places;
        return true;
    }
    void give() {
        if (device_ < 0) return;
        std::lock_guard<std::mutex> lock(mutex());
        std::multiset<int>& taken = seats()[device_];
        taken.erase(taken.find(places_));
        device_ = -1;
    }

private:
    static std::mutex& mutex() {
        static std::mutex* m = new std::mutex;  // (never destroyed: handles may outlive static objects)
        return *m;
    }
    static std::map<int, std::multiset<int>>& seats() {
        static auto* s = new std::map<int, std::multiset<int>>;
        return *s;
    }
    int device_ = -1, places_ = 0;
};

// Clusters tried in this order: a whole component in one block where it fits (63^2 in double): a sweep
// then ends with a block barrier (45 cycles) instead of a cluster barrier (500); else the largest
// cluster. A level of up to 4225 points (65^2) runs in block 0 as far as the shared memory reaches. Multigrid
// per slice on a B200 with the limits 4225, 1100 and 300: 95 x 79 89, 96, 108 us; 127^2 105, 102, 110; 160^2
// 116, 123, 138; 319^2 in single precision 197, 234, 227. 300 is for grids that fit with nothing else, and
// 8 blocks for GPUs without room for two clusters of 16.
struct ClTry { int cs, own; };
constexpr ClTry kClTries[] = {{1, 1 << 30}, {16, 4225}, {16, 1100}, {16, 300}, {8, 4225}, {8, 1100}, {8, 300}};

template <class R>
struct ClPlan {
    bool ok = false;
    ClArgs<R> a{};
    size_t smem = 0;
    int places = 0;  // clusters of this plan that an idle GPU holds

    // planes of every level for clusters of cs blocks, levels of at most `own` points in block 0
    static bool layout(ClArgs<R>& A, size_t& smem, const std::vector<MGLev>& lev, double dx, double dy, int cs,
                       int own, int ns_bottom) {
        const int nl = (int)lev.size();
        if (nl < 2 || nl > kClMaxLevels) return false;
        A = ClArgs<R>{};
        A.nl = nl;
        A.cs = cs;
        A.ns_bottom = ns_bottom;
        int nd = 0;
        for (int l = 0; l < nl; ++l) {
            ClLev<R>& L = A.lev[l];
            L.nx = lev[l].vhi_i - lev[l].vlo + 1;
            L.ny = lev[l].vhi_j - lev[l].vlo + 1;
            L.kp = (L.nx + 1) / 2;
            L.dist = l == 0 || (cs > 1 && nd == l && L.nx * L.ny > own);
            if (L.dist) nd = l + 1;
            const double f = (double)(1 << l);
            L.facx = (R)(1. / ((dx * f) * (dx * f)));
            L.facy = (R)(1. / ((dy * f) * (dy * f)));
        }
        // rows per block: even on the last split level, doubled on every finer one, so that a
        // block's coarse rows lie under its fine rows, a multiple of the rows per thread, and enough for
        // every level (a node-centred level has 2 n + 1 rows over n, one more than doubling gives where
        // the last split level fills its blocks)
        auto rows_per_thread = [&](const ClLev<R>& L, int rows) {
            const int groups = kClThreads / L.kp;
            int rt = 1;
            while (rt < 8 && groups * rt < rows) rt *= 2;
            return groups * rt < rows ? 0 : rt;
        };
        for (int l = 0; l < nl; ++l) if (A.lev[l].kp > kClThreads) return false;
        int base = cs > 1 ? 2 * ((A.lev[nd - 1].ny + 2 * cs - 1) / (2 * cs)) : 0;
        for (bool fits = cs == 1; !fits; ) {
            fits = true;
            for (int l = 0; l < nd; ++l) {
                const int rp = base << (nd - 1 - l), rt = rows_per_thread(A.lev[l], rp);
                if (!rt) return false;
                if (rp % rt || cs * rp < A.lev[l].ny) fits = false;
            }
            if (!fits) base += 2;
        }
        for (int l = 0; l < nl; ++l) {
            ClLev<R>& L = A.lev[l];
            L.rp = L.dist && cs > 1 ? base << (nd - 1 - l) : L.ny;
            L.rt = rows_per_thread(L, L.rp);
            if (!L.rt) return false;
            if (!(L.dist && cs > 1)) L.rp = (L.rp + L.rt - 1) / L.rt * L.rt;
            L.ng = L.rp / L.rt;
            L.magic = (unsigned)(((1u << 22) + L.kp - 1) / L.kp);
            L.ratio = L.facy / L.facx;
            L.nwarps = (L.kp * L.ng + 31) / 32;
        }
        // the smallest levels as one matrix: from the first level of block 0 with at most 32 storage
        // places (one point per lane of the warps that form it; a limit of 64, 7^2 instead of 3^2 on
        // 2^k - 1 grids, saved another 1 us per V-cycle and took 45 us to form)
        A.lm = nl;
        A.nm = 0;
        for (int l = nl - 1; l >= nd && l >= 1; --l) {
            const int n = A.lev[l].rp * 2 * A.lev[l].kp;
            if (n > 32 || nl - l > 6) break;
            A.lm = l;
            A.nm = n;
        }
        size_t off = 0, coff = 0;
        auto take = [&](size_t n) { const size_t o = off; off += (n + 3) / 4 * 4; return (unsigned)o; };
        auto ctake = [&](size_t n) { const size_t o = coff; coff += (n + 3) / 4 * 4; return (unsigned)o; };
        for (int l = 0; l < A.lm; ++l) {
            ClLev<R>& L = A.lev[l];
            L.inv = take((size_t)L.rp * 2 * L.kp);
            L.dia = take((size_t)L.rp * L.kp);
            if (l == 0 && std::is_same<R, float>::value) L.low = take((size_t)L.rp * 2 * L.kp);
            if (L.dist) A.dist_elems = (unsigned)off;
        }
        A.matrix = take((size_t)A.nm * A.nm);
        A.coef_elems = (unsigned)off;
        for (int l = 0; l < nl; ++l) {
            ClLev<R>& L = A.lev[l];
            const size_t row = 2 * (size_t)L.kp;
            if (l <= A.lm) {
                L.phi = take((L.rp + 2) * (row + 2));
                L.rhs = take(L.rp * row);
                L.xrow = take(L.dist && cs > 1 ? row + 2 : 0);
            }
            L.cacf = ctake(L.rp * (row + 2));
            L.cinv = ctake(L.rp * row);
            L.cxrow = ctake(L.dist && cs > 1 ? row + 2 : 0);
        }
        if (A.nm) ctake((size_t)(kClThreads / 32) * kClWarpScratch);
        A.celems = (unsigned)coff;
        // warps of the levels of block 0 do not grow on the way down
        for (int l = nl - 2; l >= nd; --l) A.lev[l].nwarps = std::max(A.lev[l].nwarps, A.lev[l + 1].nwarps);
        A.elems = (unsigned)off;
        smem = std::max(off, coff) * sizeof(R);
        return true;
    }
};

}  // namespace hpq

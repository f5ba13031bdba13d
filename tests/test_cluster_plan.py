"""The shared-memory plan of the cluster multigrid over all grids: every row of every level belongs to a
block, and the rows that the kernel reads and writes lie inside their planes. Plain C++, no GPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <cstdio>
#include <cstring>
#include "mgcl_plan.hpp"
using namespace hpq;

static long plans = 0, bad = 0;
static void fail(const char* what, int nx, int ny, int bytes, const ClTry& t, int l, long a, long b) {
    if (bad++ < 10) std::printf("%d x %d, %d bytes, cluster %d, own %d: level %d %s: %ld, %ld\n", nx, ny, bytes, t.cs, t.own, l, what, a, b);
}

template <class R>
void check(int nx, int ny) {
    const std::vector<MGLev> lev = mg_levels(nx, ny);
    for (const ClTry& t : kClTries) {
        ClArgs<R> A;
        size_t smem = 0;
        // (227 KB: the most that a block can have)
        if (!ClPlan<R>::layout(A, smem, lev, 1.0, 1.0, t.cs, t.own, mg_bottom_sweeps(lev)) || smem > 227 * 1024) continue;
        ++plans;
        const int cs = A.cs;
        auto err = [&](const char* what, int l, long a, long b) { fail(what, nx, ny, (int)sizeof(R), t, l, a, b); };
        for (int l = 0; l < A.nl; ++l) {
            const ClLev<R>& L = A.lev[l];
            const int blocks = L.dist ? cs : 1, rs = 2 * L.kp + 2;
            if ((long)blocks * L.rp < L.ny) err("rows without a block", l, (long)blocks * L.rp, L.ny);
            if (2 * L.kp < L.nx || L.rt * L.ng != L.rp || L.kp * L.ng > kClThreads) err("threads", l, L.kp, L.ng);
            for (int x = 0; x < kClThreads; ++x)
                if ((int)((x * L.magic) >> 22) != x / L.kp) err("division by kp", l, x, L.kp);
            // blocks exchange rows with a neighbour that exists, across every pair of rows of the grid
            for (int rank = 0; rank <= blocks; ++rank) {
                const bool joined = L.dist && cl_joined(rank, cs, L.rp, L.ny, nx % 2 == 0);
                if (joined && (rank == 0 || rank >= cs)) err("neighbour", l, rank, L.rp);
                if (L.dist && rank > 0 && rank * L.rp < L.ny && !joined) err("no exchange", l, rank, L.rp);
            }
            if (l <= A.lm) {
                if (L.phi + (size_t)(L.rp + 2) * rs > A.elems || L.rhs + (size_t)L.rp * 2 * L.kp > A.elems) err("plane", l, L.phi, A.elems);
                if (L.phi < A.coef_elems) err("plane in the coefficients", l, L.phi, A.coef_elems);
            }
            if (l + 1 == A.nl || l >= A.lm) continue;
            const ClLev<R>& C = A.lev[l + 1];
            if (L.dist && C.dist && cs > 1 && L.rp != 2 * C.rp) err("rows not doubled", l, L.rp, C.rp);
            // interpolation: rows of the coarse plane that the threads of every block read, in rows of that
            // block's plane, which holds rows -1 .. C.rp
            for (int rank = 0; rank < blocks; ++rank)
                for (int q = 0; q < L.rp; ++q) {
                    const int row = (L.dist ? rank * L.rp : 0) + q;
                    const int c = cl_coarse_row(row, L.dist && C.dist ? rank * (L.rp / 2) : 0, C.rp);
                    if (c - 1 < -1 || c > C.rp) err("interpolation from row", l, row, c);
                    // (a row of the block above is there if the two exchange rows of that level)
                    if (L.dist && C.dist && row < L.ny && nx % 2 && row % 2 == 0 && row > 0 && c == 0 && !cl_joined(rank, cs, C.rp, C.ny, false))
                        err("interpolation without the block above", l, row, rank);
                    // coarse rows that restriction writes
                    if (row % 2 == 0 && row / 2 < C.ny) {
                        const int d = row / 2 - (L.dist && C.dist ? rank * (L.rp / 2) : 0);
                        if (d < 0 || d >= C.rp) err("restriction to row", l, row, d);
                    }
                }
        }
    }
}

int main() {
    for (int nx = 3; nx <= 1100; ++nx)
        for (int ny = 4 - nx % 2; ny <= (nx <= 400 ? 1100 : 420); ny += 2) {
            if (mg_levels(nx, ny).size() < 2) continue;
            check<double>(nx, ny);
            check<float>(nx, ny);
        }
    // a norm keeps every bit on its way between the blocks, and is taken for another iteration's nowhere
    for (double v : {0.0, 1.0, 1.0 / 3.0, 0x1.fffffffffffffp-30, 3.141592653589793e100, 5e-324}) {
        unsigned long long b, r;
        std::memcpy(&b, &v, 8);
        for (unsigned tag : {1u, 2u, 201u, 65536u, 100001u}) {
            const ClNorm n = cl_norm(b, tag);
            r = ((unsigned long long)cl_norm_hi(n) << 32) | cl_norm_lo(n);
            if (r != b || !cl_norm_arrived(n, tag) || cl_norm_arrived(n, tag + 1) || cl_norm_arrived(ClNorm{}, tag)) ++bad, std::printf("norm %a\n", v);
            ClNorm half = n;  // (one of the two words still the older iteration's)
            half.w[1] = cl_norm(b, tag + 2).w[1];
            if (cl_norm_arrived(half, tag) || cl_norm_arrived(half, tag + 2)) ++bad, std::printf("half a norm\n");
        }
    }
    // seats: fewer solvers than the places of each of them
    {
        auto expect = [&](bool got, bool want, const char* what) { if (got != want) ++bad, std::printf("seats: %s\n", what); };
        ClSeat s[8], other, few, one;
        for (int i = 0; i < 8; ++i) expect(s[i].take(0, 7), i < 6, "seven places");
        expect(other.take(1, 7), true, "another device");
        s[2].give();
        s[2].give();
        expect(few.take(0, 3), false, "fewer places than solvers");
        expect(s[7].take(0, 7), true, "a seat given back");
        for (ClSeat& x : s) x.give();
        expect(few.take(0, 2), true, "two places, alone");
        expect(one.take(0, 148), false, "beside a solver with two places");
        { ClSeat gone; expect(gone.take(2, 2), true, "taken"); }
        expect(one.take(2, 2), true, "given back when destroyed");
    }
    std::printf("%ld plans, %ld faults\n", plans, bad);
    return bad != 0 || plans < 10000;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src = d / "check.cpp"
    src.write_text(CHECK)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "hipace2_b200", "csrc"), "-o", str(d / "check"), str(src)])
    return subprocess.run([str(d / "check")], capture_output=True, text=True)


def test_every_row_has_a_block_and_every_access_a_plane(check):
    assert check.returncode == 0, check.stdout

"""The task orders of a batch's persistent launches (xg_batch_order.h,
compiled with g++): every block once, and none before the blocks that its task
waits for -- the condition under which CTAs that take tasks in list order
cannot deadlock.  Runs without a GPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "xg_batch_order.h"
int main(int argc, char **argv)
{
    std::vector<int> n;
    for (int i = 3; i < argc; ++i) n.push_back(atoi(argv[i]));
    const auto nb = [&](int f) { return n[f]; };
    const auto cols = xg_batch_columns(atoi(argv[1]), atoi(argv[2]), nb);
    xg_batch_factor_order(cols, nb, [](int f, int I, int J) { printf("F %d %d %d 0\n", f, I, J); });
    xg_batch_backward_order(cols, [](int f, int J) { printf("B %d %d 0 0\n", f, J); });
    xg_batch_inverse_order(cols, nb, [](int f, int I, int J, int p) { printf("I %d %d %d %d\n", f, I, J, p); });
}
"""


@pytest.fixture(scope="module")
def orders(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "o.cpp").write_text(SRC)
    subprocess.run(["g++", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "exageostat_b200", "csrc"),
                    str(d / "o.cpp"), "-o", str(d / "o")], check=True)

    def run(f0, f1, nb):
        out = subprocess.run([str(d / "o"), str(f0), str(f1)] + [str(v) for v in nb], text=True, check=True,
                             capture_output=True).stdout
        lists = {"F": [], "B": [], "I": []}
        for line in out.splitlines():
            k, *v = line.split()
            lists[k].append(tuple(map(int, v)))
        return lists

    return run


@pytest.mark.parametrize("f0,nb", [(0, [1]), (0, [7]), (0, [5, 1, 9, 5, 2]), (1, [3, 8, 8, 1, 4])])
def test_orders_are_complete_and_topological(orders, f0, nb):
    lists = orders(f0, len(nb), nb)
    fields = [(f, nb[f]) for f in range(f0, len(nb))]
    seen = set()
    for f, I, J, _ in lists["F"]:  # block (I, J) of the factor
        need = {(f, I, K) for K in range(J)} | {(f, J, K) for K in range(J)} | ({(f, J, J)} if I > J else set())
        assert need <= seen and (f, I, J) not in seen
        seen.add((f, I, J))
    assert seen == {(f, I, J) for f, n in fields for J in range(n) for I in range(J, n)}
    seen = set()
    for f, J, _, _ in lists["B"]:  # block column J of the backward solve
        assert {(f, I) for I in range(J + 1, nb[f])} <= seen and (f, J) not in seen
        seen.add((f, J))
    assert seen == {(f, J) for f, n in fields for J in range(n)}
    seen, done = set(), set()
    for f, I, J, product in lists["I"]:
        if product:  # S_IJ, over L_IJ: the rows it reads, and the solves that read L_IJ
            need = {(f, I, K) for K in range(I, nb[f])} | {(f, J, K) for K in range(I, nb[f])} | \
                {(f, R, I) for R in range(J + 1)}
            assert J <= I and need <= seen and (f, I, J) not in done
            done.add((f, I, J))
        else:  # X_IJ, I <= J
            assert I <= J and {(f, I, K) for K in range(I, J)} <= seen and (f, I, J) not in seen
            seen.add((f, I, J))
    assert seen == {(f, I, J) for f, n in fields for J in range(n) for I in range(J + 1)}
    assert done == {(f, I, J) for f, n in fields for I in range(n) for J in range(I + 1)}

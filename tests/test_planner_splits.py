"""How the planner divides work: consecutive ranges of about equal cost
(even_ranges) and whole SMs per class of a batch (sm_shares), called through a
small C++ program built from csrc/layout.cpp."""
import os
import random
import subprocess

import pytest

from helpers import ROOT


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("planner") / "probe")
    csrc = os.path.join(ROOT, "hacapk_hmvm_b200", "csrc")
    subprocess.run(["/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++", "-O1", "-std=c++17", "-fopenmp",
                    "-I", csrc, "-I", os.path.join(ROOT, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "cxx", "planner_probe.cpp"), os.path.join(csrc, "layout.cpp")],
                   check=True)

    def run(lines):
        out = subprocess.run([exe], input="\n".join(lines) + "\n", capture_output=True, text=True, check=True).stdout
        return [[int(v) for v in row.split()] for row in out.strip().split("\n")]

    return run


def _least_cap(cost, n):
    """The smallest largest range of n consecutive ranges (dynamic bisection over all sums)."""
    lo, hi = max(cost), sum(cost)
    while lo < hi:
        mid, used, acc = (lo + hi) // 2, 1, 0
        for c in cost:
            if acc + c > mid:
                used, acc = used + 1, 0
            acc += c
        lo, hi = (lo, mid) if used <= n else (mid + 1, hi)
    return lo


def test_even_ranges(planner):
    rng = random.Random(5)
    cases = [(1, [7]), (5, [3]), (4, []), (3, [1, 1, 1]), (3, [9, 1, 1, 1, 9]), (2, [0, 0, 5, 0])]
    cases += [(rng.randint(1, 40), [rng.randint(0, 10 ** rng.randint(1, 6)) for _ in range(rng.randint(1, 200))])
              for _ in range(150)]
    for (n, cost), b in zip(cases, planner([f"ranges {n} " + " ".join(map(str, c)) for n, c in cases])):
        assert len(b) == n + 1 and b[0] == 0 and b[-1] == len(cost) and b == sorted(b), (n, cost, b)
        if cost:
            largest = max(sum(cost[i:j]) for i, j in zip(b, b[1:]))
            assert largest <= _least_cap(cost, n) + sum(cost) // n // 1024 + 1, (n, cost, b)


def test_sm_shares_fit_the_gpu(planner):
    """No more SMs than there are, also where several classes want less than one."""
    rng = random.Random(6)
    cases = [(148, [(0.30, 1), (0.44, 1), (147.26, 1)]), (148, [(1, 1)] * 3), (148, [(0.1, 1)] * 10 + [(900, 2)]),
             (4, [(1, 1), (1, 1), (50, 1), (60, 1)]), (148, [(1e-3, 7), (5, 9), (5, 9)]), (148, [(3, 1)])]
    for _ in range(300):
        k = rng.randint(1, 12)
        cases.append((148, [(10 ** rng.uniform(-3, 3), rng.randint(1, 6)) for _ in range(k)]))
    lines = [f"shares {s} {len(c)} " + " ".join(f"{w!r} {p}" for w, p in c) for s, c in cases]
    for (sms, classes), share in zip(cases, planner(lines)):
        assert min(share) >= 1
        assert sum(s * p for s, (_, p) in zip(share, classes)) <= sms, (sms, classes, share)
        total = sum(w * p for w, p in classes)
        for s, (w, p) in zip(share, classes):  # nobody far above its part of the work
            assert s <= max(1, sms * w / total + 1), (sms, classes, share)


def test_sm_shares_with_more_passes_than_sms(planner):
    assert planner(["shares 4 3 1 2 100 3 1 1"]) == [[1, 1, 1]]

"""How the attention of a sampled step is cut (sample_split.h), on the CPU: every position in a slice, no more slices than the
partials' buffers hold, one wave of CTAs where that is possible, and a new cut (a graph of its own) every 16 steps at most."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def cuts(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("sample_split") / "check")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "rustane_b200", "csrc"),
                           os.path.join(ROOT, "tests", "kernels", "sample_split_check.cpp"), "-o", exe])

    def run(*args):
        lines = subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, check=True).stdout.split("\n")[:-1]
        return [tuple(int(x) for x in line.split()) for line in lines[:-1]], tuple(int(x) for x in lines[-1].split())

    return run


@pytest.mark.parametrize("shared,first,steps,gqa,samples,kv,most", [
    (1024, 1, 200, 1, 8, 32, 32),     # the benchmark's 5B decoder
    (960, 41, 200, 1, 8, 32, 32),
    (0, 5, 256, 1, 16, 32, 32),       # no shared page
    (2880, 1, 500, 4, 8, 4, 32),
    (64, 1, 60, 1, 8, 4, 2),          # two pages: one slice of each kind
    (0, 3, 60, 8, 2, 1, 1),           # one page
    (3968, 1, 120, 16, 16, 8, 32),    # more blocks than a wave of CTAs
    (256, 16, 100, 3, 11, 8, 32),
])
def test_cuts_of_a_sampled_loop(cuts, shared, first, steps, gqa, samples, kv, most):
    rows, (blocks, per_block) = cuts(shared, first, steps, gqa, samples, kv, most, 148)
    for k, (_, rounds, spans, ns, own) in enumerate(rows):
        assert ns * rounds * 64 >= shared and own * spans * 16 >= first + k
        assert (shared == 0) == (ns == 0) and own >= 1 and ns + own <= most
        if kv * blocks * 2 <= 3 * 148:
            assert kv * blocks * (ns + own) <= 3 * 148
        tasks = spans * min(per_block, samples)
        assert tasks <= 4 * max(rounds, min(per_block, samples))  # a warp's turns
    assert len({r[0] for r in rows}) <= steps // 16 + 2

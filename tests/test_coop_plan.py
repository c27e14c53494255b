"""The rule of the solver's persistent cycle (coop_plan.h), on the CPU: a device
without cooperative launches never takes it, every plan covers its nodes with one
CTA per SM at most, and its shared memory fits up to the largest restart."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SMEM = 232448 - 512  # 227 KB less the kernel's static part


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("coop") / "coop_plan_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", exe, os.path.join(HERE, "cpp", "coop_plan_check.cpp")], check=True)

    def ask(rows):
        text = "\n".join(" ".join(str(int(v)) for v in r) for r in rows)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split()
        return [tuple(int(v) for v in out[i:i + 4]) for i in range(0, len(out), 4)]

    return ask


SIZES = sorted({1, 7, 8, 9, 1215, 1216, 1217} | {int(1.07 ** k) for k in range(1, 200)} | set(range(136000, 137600, 97)))
FORMS = [(f, s) for f in (0, 1) for s in (0, 1)]


def test_without_cooperative_launches_the_separate_kernels_run(plans):
    assert not any(p[0] for p in plans([(0, 152, SMEM, N, f, s, 100) for N in SIZES for f, s in FORMS]))


@pytest.mark.parametrize("sms", [1, 76, 132, 152])
def test_plans_cover_the_nodes_and_fit(plans, sms):
    ask = [(1, sms, SMEM, N, f, s, m) for N in SIZES for f, s in FORMS for m in (1, 255)]
    taken = 0
    for (_, _, _, N, f, s, m), (planned, chunk, grid, fixed) in zip(ask, plans(ask)):
        if not planned:
            assert N > 900 * sms
            continue
        taken += 1
        assert chunk % 8 == 0 and 1 <= grid <= sms
        assert (grid - 1) * chunk < N <= grid * chunk
        assert fixed <= SMEM
    assert taken

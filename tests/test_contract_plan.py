"""Block sizes, K ranges and scratch of kpm_2d's contraction
(kpmgb_contract_plan.h), compiled with g++ into a small driver: every block of a
call fits the scratch sized for its largest, and blocks chosen from a budget
leave that scratch its place (the FP64 kernel's few MB aside)."""
import random
import shutil
import subprocess
from pathlib import Path

import pytest

from kpm_gb300 import kpm_2d_blocking

ROOT = Path(__file__).resolve().parents[1]
GIB = 1 << 30


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("plan") / "plan_driver"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{ROOT / 'kpm.jl_gb300' / 'csrc'}",
                    str(ROOT / "tests" / "contract_plan_driver.cpp"), "-o", str(exe)], check=True)

    def run(calls):
        text = "\n".join(" ".join(map(str, (*c, 152))) for c in calls)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True)
        return [tuple(map(int, line.split())) for line in out.stdout.splitlines()]
    return run


def _calls(n, seed, fixed):
    rng = random.Random(seed)
    calls = [(885016, 512, 355, 16, GIB, 0), (1 << 20, 512, 320, 512, GIB, 0),
             (1 << 20, 512, 320, 16, GIB, 0)] if fixed else []
    while len(calls) < n:
        K = int(2 ** rng.uniform(8, 23))
        NC = rng.randint(2, 700)
        arr = rng.randint(2, NC + 3) if fixed else 0
        right = rng.randint(1, NC + 3) if fixed or rng.random() < 0.3 else 0
        budget = int(2 ** rng.uniform(16, 37))
        calls.append((K, NC, arr, right, budget, int(rng.random() < 0.2)))
    return calls


def test_every_block_fits(plan):
    calls = _calls(4000, 1, True) + _calls(4000, 2, False)
    for c, (KL, KR, _, scratch, largest, _) in zip(calls, plan(calls)):
        assert largest <= scratch, c


def test_explicit_blocks_take_the_planes(plan):
    calls = _calls(2000, 3, True)
    for c, (KL, KR, k_range, *_) in zip(calls, plan(calls)):
        assert (KL, KR) == (c[2], c[3]), c
        assert (k_range > 0) == (not c[5]), c


def test_budget(plan):
    calls = _calls(6000, 4, False)
    planes = 0
    for c, (KL, KR, k_range, scratch, _, fp64) in zip(calls, plan(calls)):
        K, NC, arr, right, budget, split = c
        block = 16 * K
        kw = dict(workspace_bytes=budget, right_block=right or "auto")
        if KL == 0:   # refused: so does the reference's rule
            with pytest.raises(ValueError):
                kpm_2d_blocking(K, 1, NC, **kw)
            continue
        held = (min(KL, NC) + min(KR, NC) + 4) * block
        planes += k_range > 0
        assert scratch <= max(budget - held, fp64), c
        if min(KL, NC) < NC:
            # a blocked call follows the rule up to a third for the planes
            rule = kpm_2d_blocking(K, 1, NC, **kw)["arr_size"]
            assert 2 * rule <= 3 * KL and KL <= rule, c
    assert planes > len(calls) // 4


@pytest.mark.parametrize("K,NC", [(16384 * 4, 64), (8192 * 27, 64), (131072 * 16, 512)])
def test_no_budget_takes_the_planes(plan, K, NC):
    (KL, KR, k_range, *_), = plan([(K, NC, 0, 0, 100 * GIB, 0)])
    assert KL == KR == NC and k_range > 0


@pytest.mark.parametrize("K", [1 << 20, 131072 * 16])
def test_blocked_call_keeps_the_planes(plan, K):
    """A budget that holds a part of the left block leaves the planes theirs."""
    (KL, KR, k_range, *_), = plan([(K, 512, 0, 0, 4 * GIB, 0)])
    assert 2 <= KL < 512 and k_range > 0

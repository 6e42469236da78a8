"""The bounce planned for the path-finishing launch comes from queue lengths that the iteration recorded."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "tail_plan")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-ffp-contract=off", f"-I{cuda}/include", os.path.join(ROOT, "tests", "cpp", "tail_plan.cpp"),
                    "-o", exe], check=True, capture_output=True)

    def run(queues, max_bounces=8, first=2, tail_paths=98304, nee=1, cost=1, launched=-1, keep=-1):
        many = isinstance(queues[0], list)
        lines = [" ".join(str(x) for x in (max_bounces, first, tail_paths, nee, cost, launched, keep, len(q), *q))
                 for q in (queues if many else [queues])]
        out = subprocess.run([exe], input="\n".join(lines), check=True, capture_output=True, text=True).stdout.split()
        return [int(x) for x in out] if many else int(out[0])

    return run


SHORT = [1_000_000, 300_000, 1500, 90, 5, 0, 0]  # pays from bounce 2 on
LONG = [1_000_000, 900_000, 800_000, 700_000, 600_000, 500_000, 400_000]


def test_device_decided_iteration(plan):
    assert plan(SHORT) == 2
    assert plan(SHORT, first=4) == 4
    assert plan(SHORT, tail_paths=100) == 3
    assert plan(LONG) == 8                       # no tail
    assert plan(LONG, tail_paths=-1) == 8
    assert plan([5, 0, 0, 0], first=0, tail_paths=0) == 1  # an empty queue: nothing is launched after it


# a planned iteration records the bounces up to its hand-over; what follows them reads as zero
@pytest.mark.parametrize("launched", [0, 1, 2, 3, 5])
def test_unrecorded_lengths_are_not_empty_queues(plan, launched):
    recorded = LONG[:launched + 1]
    assert plan(recorded, launched=launched, keep=launched) == -1
    assert plan(recorded, launched=launched, keep=-1) == -1
    paying = LONG[:launched] + [700]
    assert plan(paying, launched=launched, first=0, keep=launched) == launched


def test_a_plan_without_tail_has_every_length(plan):
    assert plan(LONG, launched=8) == 8
    assert plan([1_000_000, 300_000, 200_000, 100_000, 50, 3, 0], launched=8) == 4


def test_a_plan_stays_near_the_line(plan):
    at = 1 + plan([[10 * q, 2 * q, q] for q in range(1, 98304)], launched=2).index(-1)
    assert plan([10 * at, 2 * at, at], launched=2, keep=2) == 2
    assert plan([10 * at, 2 * at, at], launched=2, keep=1) == -1


def test_without_the_cost_rule_only_the_length_counts(plan):
    assert plan(LONG, cost=0, tail_paths=800_000) == 2
    assert plan(LONG, cost=0, tail_paths=600_000) == 4
    assert plan(LONG, cost=0, first=0, tail_paths=1 << 30) == 0
    assert plan(LONG[:4], cost=0, tail_paths=98304, launched=3) == -1

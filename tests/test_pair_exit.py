"""The rules by which two CTAs that share a ring of operand slots may end, played through on the host: nothing may still be on its
way into the shared memory of a CTA that has ended, in whatever order copies and commits arrive and wherever a role gave up."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("needs a C++ compiler")
    exe = tmp_path_factory.mktemp("pair_exit") / "model"
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", str(ROOT / "torchpairwise_b200" / "csrc"), str(ROOT / "tests" / "pair_exit_model.cpp"),
                    "-o", str(exe)], check=True)
    return lambda *args: [int(v) for v in subprocess.run([str(exe), *args], check=True, capture_output=True, text=True).stdout.split()]


def test_nothing_is_under_way_when_a_pair_ends(model):
    runs, gave_up, early, stuck = model("20000")
    assert runs == 20000 and runs // 5 < gave_up < runs
    assert early == 0, "an arrival was under way into shared memory that had been given up"
    assert stuck == 0, "a wait at the end had nothing to complete it"


def test_the_model_sees_an_end_that_waits_for_accumulators_alone(model):
    """As the kernels once ended: the last accumulators were waited for, the commits that release slots and, after an error, the
    copies of the other CTA were not."""
    runs, _, early, _ = model("2000", "unwaited")
    assert early > runs // 4

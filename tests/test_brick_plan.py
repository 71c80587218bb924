"""The brick planner on the CPU: tests/native/brick_plan_check.cpp runs its tables as the kernels would."""
import subprocess
from pathlib import Path

import pytest

from genesis_tissue_simulation_gb300 import build as native_build

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    program = tmp_path_factory.mktemp("plan") / "brick_plan_check"
    cuda = Path(native_build.nvcc_path()).resolve().parents[1]
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{cuda / 'include'}", f"-I{native_build.CSRC}", "-o", str(program),
                    str(ROOT / "tests" / "native" / "brick_plan_check.cpp"), str(native_build.CSRC / "brick_plan.cpp"), "-lpthread"], check=True)

    def run(size, holes=0, forced=0, local=8000, whole=False, reverse=False, passes=0):
        args = [*size, holes, forced, local, int(whole), int(reverse), passes]
        result = subprocess.run([str(program), *map(str, args)], capture_output=True, text=True)
        assert result.returncode == 0, (args, result.stdout)
        return tuple(int(v) for v in result.stdout.split())
    return run


@pytest.mark.parametrize("size,holes,counts", [((1, 1, 1), 0, (0,)), ((3, 3, 3), 0, (0, 2, 30)), ((2, 9, 2), 0, (0, 7, 152)), ((64, 3, 3), 0, (0, 152)),
                                               ((10, 9, 6), 100, (1, 7, 30)), ((16, 8, 16), 0, (0, 5, 60)), ((23, 13, 19), 50, (0,)), ((40, 20, 30), 0, (0,))])
@pytest.mark.parametrize("kind", [dict(), dict(whole=True), dict(reverse=True), dict(whole=True, passes=1)], ids=["plain", "damped", "reverse", "guard"])
def test_bricks_sweep_as_the_whole_mesh_does(check, size, holes, counts, kind):
    for forced in counts:
        bricks, stages = check(size, holes, forced, **kind)
        assert bricks >= 1 and (forced != 1 or bricks == 1)


def test_meshes_that_do_not_fit_have_no_plan(check):
    assert check((16, 8, 16), local=10)[0] == 0          # more nodes than the bricks hold
    assert check((16, 8, 16), local=150)[0] == 0         # the nodes fit, the halo does not
    assert check((16, 8, 16), forced=1, local=2000)[0] == 0

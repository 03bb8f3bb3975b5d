"""The warp roles of the attention kernels under adversarial schedules, on the CPU.

``tests/schedules`` compiles the kernel sources as they are with a host compiler: barriers, copies and
the tensor pipe are simulated, arithmetic and data movement are left out, and the order in which warps go
on is drawn at random with some of them held back for long.  No schedule may deadlock, let a warp
arrive twice in one phase of a barrier, or let a wait return on a phase that it has already seen; and no
warp may read global memory before it has waited for the kernel before its own.
"""

import re
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "flash_attention_triton_b200" / "csrc"


@pytest.fixture(scope="module")
def simulator(tmp_path_factory):
    build = tmp_path_factory.mktemp("schedules")
    for source in (*(CSRC / n for n in ("common.cuh", "mma_issue.cuh", "bwd_roles.cuh", "bwd.cu", "fwd.cu")),
                   *(HERE / "schedules").iterdir()):
        shutil.copy(source, build)
    for stand_in in ("cuda.h", "ptx.cuh"):
        (build / stand_in).write_text('#include "cuda_runtime.h"\n')
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I.", "main.cpp", "-o", "simulator"], cwd=build, check=True,
                   capture_output=True, text=True)
    return build / "simulator"


def check(simulator, kernel, headdim, rows, keys, steps=(128,), schedules=60):
    for step in steps:
        run = subprocess.run([simulator, kernel, str(headdim), str(rows), str(keys), str(schedules), str(step)],
                             capture_output=True, text=True, timeout=300)
        assert run.returncode == 0, (step, run.stdout + run.stderr)


def steps_of(headdim):
    return (64, 128) if headdim <= 64 else (128,)


def test_no_kernel_takes_the_read_only_path_to_global_memory():
    """A kernel starts while the one before it still writes: what it reads must neither come through the
    non-coherent path nor be open to the compiler's use of it (const __restrict__ parameters)."""
    for source in CSRC.glob("*.cu*"):
        if source.name == "selftest.cu":  # an ordinary launch
            continue
        code = re.sub(r"//.*", "", source.read_text())
        assert not re.search(r"__ldg|\.nc\b|const \w+\* ?__restrict__", code), source.name


@pytest.mark.parametrize("rows,keys", [(1, 1), (128, 64), (449, 300), (640, 640)])
@pytest.mark.parametrize("kernel", ["dkdv", "dkdv_atomic", "dkdv_spill"])
@pytest.mark.parametrize("headdim", [32, 64, 96, 128])
def test_dk_dv_roles(simulator, kernel, headdim, rows, keys):
    check(simulator, kernel, headdim, rows, keys, (128,) if kernel == "dkdv_spill" else steps_of(headdim))


@pytest.mark.parametrize("rows,keys", [(1, 1), (128, 64), (449, 300), (640, 640)])
@pytest.mark.parametrize("headdim", [32, 64, 96, 128])
def test_dq_roles(simulator, headdim, rows, keys):
    check(simulator, "dq", headdim, rows, keys, steps_of(headdim))


@pytest.mark.parametrize("rows,keys", [(1, 1), (128, 64), (449, 300), (1200, 1200)])
@pytest.mark.parametrize("headdim", [32, 64, 96, 128, 256])
def test_forward_roles(simulator, headdim, rows, keys):
    """One CTA takes every work item: what an item leaves on its way to a barrier meets the next one."""
    check(simulator, "fwd", headdim, rows, keys, steps_of(headdim))


@pytest.mark.parametrize("rows,keys", [(700, 300), (1200, 1200), (2200, 1000)])
@pytest.mark.parametrize("headdim", [32, 64])
def test_forward_roles_single_tile_items_one_after_the_other(simulator, headdim, rows, keys):
    """So few SMs that a CTA takes several items of one Q tile each: the softmax group without a tile has nothing to
    wait for and must not run ahead of the other one."""
    tiles = (rows + 127) // 128
    sms = (2 * tiles + 6) // 7  # fwd_tiles_per_item: the fewest that give single-tile items
    assert tiles > 2 * sms
    run = subprocess.run([simulator, "fwd", str(headdim), str(rows), str(keys), "60", "64", str(sms)],
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout + run.stderr


@pytest.mark.parametrize("rows,keys", [(1, 1), (128, 64), (449, 300), (640, 640)])
@pytest.mark.parametrize("kernel,headdim", [("scores", 256), ("consume", 64), ("consume", 128), ("consume", 256),
                                            ("consume_pair", 256)])
def test_spill_roles(simulator, kernel, headdim, rows, keys):
    check(simulator, kernel, headdim, rows, keys)


@pytest.mark.parametrize("kernel", ["scores", "consume", "consume_pair", "fwd"])
def test_roles_of_three_chunk_heads(simulator, kernel):
    check(simulator, kernel, 192, 449, 300)
    check(simulator, kernel, 192, 640, 640)


@pytest.mark.parametrize("rows,keys", [(128, 64), (449, 300), (1200, 1200)])
@pytest.mark.parametrize("headdim", [32, 64, 96, 128, 192, 256])
def test_forward_that_gives_up_a_wait(simulator, headdim, rows, keys):
    """Whichever wait runs into its limit, every CTA ends and the work counter is at zero for the next launch."""
    for step in steps_of(headdim):
        for sms in (1, 2, 3, 64):
            run = subprocess.run([simulator, "fwd", str(headdim), str(rows), str(keys), "60", str(step), str(sms), "giveup"],
                                 capture_output=True, text=True, timeout=300)
            assert run.returncode == 0, (step, sms, run.stdout + run.stderr)


@pytest.mark.parametrize("kernel,headdim", [("dkdv", 64), ("dkdv", 128), ("dkdv_atomic", 32), ("dkdv_atomic", 128), ("dkdv_spill", 128),
                                            ("dq", 64), ("dq", 128), ("scores", 192), ("scores", 256), ("consume", 128),
                                            ("consume", 256), ("consume_pair", 256)])
def test_backward_that_gives_up_a_wait(simulator, kernel, headdim):
    for step in steps_of(headdim):
        for rows, keys in ((128, 64), (640, 640)):
            run = subprocess.run([simulator, kernel, str(headdim), str(rows), str(keys), "60", str(step), "1", "giveup"],
                                 capture_output=True, text=True, timeout=300)
            assert run.returncode == 0, (step, rows, run.stdout + run.stderr)


@pytest.mark.parametrize("headdim,step", [(64, 64), (64, 128), (128, 128), (256, 128)])
@pytest.mark.parametrize("sms", [2, 5, 64])
def test_forward_items_go_heaviest_first_to_whichever_cta_runs(simulator, headdim, step, sms):
    """The simulator runs CTAs one after the other, like CTAs of a launch that find an SM late: none of them may have
    kept an item heavier than those that others have done by then."""
    run = subprocess.run([simulator, "fwd", str(headdim), "2900", "2900", "20", str(step), str(sms), "order"],
                         capture_output=True, text=True, timeout=300, check=True)
    for line in run.stdout.splitlines():
        items = list(dict.fromkeys(int(row) // 256 for row in line.split()))  # pairs of Q tiles, at their first store
        assert items == sorted(items, reverse=True) and len(items) == 12

"""Host-side mirror of the reference interface: names, defaults, config shim, partitioning."""

from __future__ import annotations

import inspect
import os
import subprocess
import sys
import textwrap

import pytest
import torch

import flash_attention_triton_b200 as fa
from conftest import ROOT
from flash_attention_triton_b200 import shard_range, shard_slab


def test_public_names_match_reference_package():
    # the reference exports exactly these four (src/flash_attention_triton/__init__.py:13)
    for name in ("KernelsConfigV2", "flash_attention_v2", "flash_attention_v2_custom", "init_to_zero_v2"):
        assert hasattr(fa, name)


def test_flash_attention_v2_signature():
    sig = inspect.signature(fa.flash_attention_v2)
    assert list(sig.parameters) == ["q", "k", "v", "softmax_scale", "deterministic"]
    assert sig.parameters["softmax_scale"].default is None
    assert sig.parameters["deterministic"].default is False
    sig = inspect.signature(fa.flash_attention_v2_custom)
    assert list(sig.parameters) == ["q", "k", "v", "softmax_scale", "kernels_configs"]


def test_cpu_tensors_are_rejected_like_the_reference():
    q = torch.randn(1, 1, 16, 32)
    with pytest.raises(AssertionError, match="CUDA"):
        fa.flash_attention_v2(q, q, q)


class _Cfg:
    def __init__(self, **kw):
        self.kwargs = kw


def test_config_shim_maps_sequence_parallel_to_determinism():
    mk = lambda seqpar: fa.KernelsConfigV2(128, 128, 32, 256, 32, 8, 16, 1, [
        _Cfg(BLOCK_Q_ROWS_SIZE=64, BLOCK_KV_COLS_SIZE=64, SEQUENCE_PARALLEL=seqpar)])
    assert mk(False).is_deterministic() is True
    assert mk(True).is_deterministic() is False
    with pytest.raises(Exception):
        mk(True).block_rows_size = 1  # frozen, like the reference dataclass


def test_init_to_zero_v2_zeroes_named_tensor():
    t = torch.ones(4)
    out = fa.init_to_zero_v2("DQ")({"DQ": t})
    assert out is t and torch.equal(t, torch.zeros(4))


@pytest.mark.parametrize("n,world", [(64, 1), (64, 2), (64, 8), (16, 8), (10, 4), (3, 8), (0, 2)])
def test_shard_ranges_partition_the_batch_head_axis(n, world):
    ranges = [shard_range(n, world, r) for r in range(world)]
    assert ranges[0][0] == 0 and ranges[-1][1] == n
    for (a0, a1), (b0, b1) in zip(ranges, ranges[1:]):
        assert a1 == b0
    sizes = [b - a for a, b in ranges]
    assert max(sizes) - min(sizes) <= 1


def test_shard_range_rejects_bad_rank():
    with pytest.raises(ValueError):
        shard_range(8, 2, 2)
    with pytest.raises(ValueError):
        shard_range(8, 0, 0)


def test_shard_slab_is_a_view_of_contiguous_heads():
    t = torch.arange(2 * 4 * 3 * 2, dtype=torch.float32).view(2, 4, 3, 2)
    parts = [shard_slab(t, 4, r) for r in range(4)]
    assert all(p.shape == (1, 2, 3, 2) for p in parts)
    torch.testing.assert_close(torch.cat(parts, dim=1).view(2, 4, 3, 2), t)


GLOO_WORKER = textwrap.dedent(
    """
    import os, sys, torch, torch.distributed as dist
    sys.path.insert(0, os.environ["FA2_ROOT"])
    from flash_attention_triton_b200 import shard_slab, shard_range
    from oracle.attention_oracle import naive_attention
    dist.init_process_group("gloo")
    rank, world = dist.get_rank(), dist.get_world_size()
    g = torch.Generator().manual_seed(0)
    q, k, v, do = (torch.randn(2, 3, 40, 16, generator=g) for _ in range(4))
    mine = [shard_slab(t, world, rank) for t in (q, k, v, do)]
    r = naive_attention(*mine, dtype=torch.float32)
    # gather the per-rank slabs on rank 0 and compare with the unsharded computation
    for key in ("o", "dq", "dk", "dv"):
        parts = [None] * world
        dist.all_gather_object(parts, r[key])
        if rank == 0:
            full = naive_attention(q, k, v, do, dtype=torch.float32)[key].reshape(1, 6, 40, 16)
            assert torch.equal(torch.cat(parts, dim=1), full), key
    dist.barrier()
    dist.destroy_process_group()
    """
)


def test_two_ranks_cover_the_problem_without_a_collective_on_the_data_path(tmp_path):
    """world_size-2 gloo run: each rank computes its own (batch, head) slab with the oracle;
    the concatenation equals the unsharded result bit for bit."""
    script = tmp_path / "worker.py"
    script.write_text(GLOO_WORKER)
    env = dict(os.environ, FA2_ROOT=str(ROOT), OMP_NUM_THREADS="2")
    res = subprocess.run(
        [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2",
         "--master-addr", "127.0.0.1", "--master-port", "29511", str(script)],
        env=env, capture_output=True, text=True, timeout=240,
    )
    assert res.returncode == 0, res.stderr[-2000:]


def _readable_by_definition(t):
    """Unit last stride, 16-byte aligned base, positive batch / head / row strides in multiples of 8
    elements where the dimension has more than one entry, rows that do not overlap."""
    if t.stride(-1) != 1 or t.data_ptr() % 16:
        return False
    if any(n > 1 and (s <= 0 or s % 8) for n, s in zip(t.shape[:3], t.stride()[:3])):
        return False
    return t.shape[2] == 1 or t.stride(2) >= t.shape[3]


@pytest.mark.parametrize("base", [torch.zeros(4096, dtype=torch.float16), torch.zeros(4096, dtype=torch.bfloat16)])
def test_native_host_path_takes_the_same_tensors_in_place(base):
    from flash_attention_triton_b200 import _lib

    shapes = [(2, 3, 4, 16), (1, 3, 4, 16), (2, 1, 4, 16), (2, 3, 1, 16), (1, 1, 1, 8)]
    strides = [(192, 64, 16, 1), (192, 16, 48, 1), (0, 64, 16, 1), (64, 0, 16, 1), (192, 60, 16, 1),
               (196, 64, 16, 1), (192, 64, 8, 1), (192, 64, 20, 1), (192, 64, 16, 2), (192, 1, 16, 4), (5, 3, 7, 1)]
    seen = set()
    for shape in shapes:
        for stride in strides:
            for offset in (0, 1, 8):
                t = base.as_strided(shape, stride, offset)
                want = _readable_by_definition(t)
                seen.add(want)
                assert _lib.host().readable_in_place(t) is want, (shape, stride, offset)
    assert seen == {True, False}


def test_native_host_path_refuses_what_is_not_a_tensor():
    from flash_attention_triton_b200 import _lib

    t = torch.zeros(1, 1, 8, 8, dtype=torch.float16)
    for call in (lambda h: h.forward(t, t, None, 0.1, False), lambda h: h.forward(t, t, t),
                 lambda h: h.forward(t, t, t, "x", False), lambda h: h.gradients(t, 1, t, False), lambda h: h.preprocess(t, t[0, 0], t), lambda h: h.readable_in_place(2),
                 lambda h: h.backward(*([t] * 7), None, None, 0.1, 0), lambda h: h.backward(t)):
        with pytest.raises(TypeError):
            call(_lib.host())


def test_status_check_reads_the_word_of_the_tensors_device(monkeypatch):
    """Tensors on cuda:1 while cuda:0 is current, on a fake library: the word read, and reported, is cuda:1's."""
    from contextlib import contextmanager
    from types import SimpleNamespace

    from flash_attention_triton_b200 import _lib, api

    current = [torch.device("cuda:0")]

    @contextmanager
    def device(d):
        current.append(d)
        yield
        current.pop()

    words = {torch.device("cuda:0"): 0, torch.device("cuda:1"): 0x10003}
    fake = SimpleNamespace(forward=lambda *a: (0, "o", "lse", None), readable_in_place=lambda t: True,
                           preprocess=lambda o, do, lse: (0, "rowstats", do), backward=lambda *a: 0)
    monkeypatch.setattr(_lib, "host", lambda: fake)
    monkeypatch.setattr(_lib, "device_status", lambda: words[current[-1]])
    monkeypatch.setattr(torch.cuda, "device", device)
    t = SimpleNamespace(shape=torch.Size((1, 2, 8, 64)), dtype=torch.float16, is_cuda=True,
                        device=torch.device("cuda:1"), is_contiguous=lambda: True)
    lse = SimpleNamespace(shape=torch.Size((1, 2, 8)))
    calls = (lambda: api._flash_attention_forward(t, t, t, None),
             lambda: api._flash_attention_backward(t, t, t, t, lse, t, t, t, t, 0.1, True))
    for call in calls:
        call()  # not asked: not read
    monkeypatch.setenv("FA2_B200_CHECK_STATUS", "1")
    for call in calls:
        with pytest.raises(_lib.Fa2Error, match="0x10003"):
            call()


def test_host_module_is_rebuilt_for_another_torch(monkeypatch, tmp_path):
    from types import SimpleNamespace

    from flash_attention_triton_b200 import build

    runs = []

    def compile_(cmd, **kwargs):
        runs.append(cmd)
        (tmp_path / "_host.so").touch()
        return SimpleNamespace(returncode=0)

    monkeypatch.setattr(build, "HOST_PATH", tmp_path / "_host.so")
    monkeypatch.setattr(build, "BUILD_DIR", tmp_path)
    monkeypatch.setattr(build.subprocess, "run", compile_)
    for version, expected in (("1", 1), ("1", 1), ("2", 2), ("2", 2)):
        monkeypatch.setattr(torch, "__version__", version)
        build._build_host(False)
        assert len(runs) == expected


def test_native_call_leaves_cpu_tensors_to_the_general_path():
    """What it refuses of CUDA tensors: test_native_call_serves_plain_tensors_only in test_gpu_parity.py."""
    from flash_attention_triton_b200 import _lib

    attention = _lib.host().attention
    t = torch.zeros(1, 2, 8, 16, dtype=torch.float16)
    assert attention(t, t, t, None, False) is None
    assert attention(t, t, 3, None, False) is None
    with pytest.raises(TypeError):
        attention(t, t, t)


def test_one_rule_and_one_ladder_for_native_and_python_calls(monkeypatch):
    """api.py asks the native module, so the tests of its functions test what plain calls do; sizes where the rule changes."""
    from flash_attention_triton_b200 import _lib, api

    monkeypatch.delenv("FA2_B200_BWD_MODE", raising=False)
    host = _lib.host()
    for n in (1, 128, 8192, 46208, 46209, 65536):  # 361 tiles: 65 341 pairs of 32 KiB, below 2 GiB; 362: above
        for d in (8, 64, 72, 128, 136, 256):
            for det in (False, True):
                spill = d > 128 or (d > 64 and n <= 46208)
                want = api._MODE_SPILL if spill else api._MODE_RECOMPUTE if det or d > 64 else api._MODE_ATOMIC
                assert host.backward_mode(det, d, n) == want == api._backward_mode(det, d, n)
    head = 2080 * 32768

    def ladder(limit, d, mode):
        asked = []
        take = lambda size: asked.append(size) or (torch.zeros(1) if size <= limit else None)
        return *host.allocate_workspace(take, 2, 32, 8192, d, mode)[1:], asked

    assert ladder(1 << 62, 128, 2) == (32 * head, 2, [32 * head])
    assert ladder(4 * head, 128, 2) == (4 * head, 2, [32 * head, 4 * head])
    assert ladder(head, 128, 2) == (head, 2, [32 * head, 4 * head, head])
    assert ladder(0, 128, 2) == (0, 1, [32 * head, 4 * head, head])
    assert ladder(0, 128, 1) == (0, 1, [])
    assert ladder(0, 64, 0)[1] == -1 and len(ladder(0, 64, 0)[2]) == 1  # the accumulator of the atomic mode is a need
    assert ladder(0, 256, 2)[1] == -1
    with pytest.raises(ZeroDivisionError):
        host.allocate_workspace(lambda size: 1 / 0, 2, 32, 8192, 128, 2)
    with pytest.raises(TypeError):
        host.allocate_workspace(lambda size: 3, 2, 32, 8192, 128, 2)

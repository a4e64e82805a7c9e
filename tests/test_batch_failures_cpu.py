"""A batch whose tile configuration cannot be changed: one that does not fit leaves the batch as
it was (runs, and replays of its captured graph, go on); one whose buffers cannot be had leaves it
without a plan, so that no kernel is launched on buffers that are gone, until another is set.
On the CPU, with a stand-in for the CUDA runtime whose allocations can be made to fail."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SCRIPT = """
import ctypes, sys
sys.path.insert(0, {root!r})
from ctypes import byref, c_int, c_void_p
from fasterbackprojection_gb300 import _lib, make_info
from fasterbackprojection_gb300._lib import CaptureDesc
lib, fake = _lib.load(), ctypes.CDLL(None)
ctx, batch, stream = c_void_p(), c_void_p(), c_void_p(1)
_lib.check(lib.fbp_create(byref(ctx), 0))
wide = {wide}
# Tiles of configuration 2 reach twice as far along the second axis as those of 0 and 1.
infos = [make_info(num_laser_targets=64, num_time_bins=40000, time_step=1e-3, voxel_res=(32, 32, 32),
                   hidden_min=(-1, -2, -1), voxel_size=(0.01, 0.01, 0.45 if wide and not k else 0.1)) for k in range(2)]
caps = (CaptureDesc * 2)()
for k, info in enumerate(infos):
    caps[k].info, caps[k].cube, caps[k].laser_xyz, caps[k].volume = info, 4096, 4096, 4096
    caps[k].dtype, caps[k].layout = 0, 1
_lib.check(lib.fbp_batch_create(ctx, 2, caps, byref(batch)))

def run(graph):
    a, g = fake.fake_launches(), fake.fake_graph_launches()
    st = lib.fbp_batch_run(batch, graph, stream)
    return st, fake.fake_launches() - a, fake.fake_graph_launches() - g

first = run(0)
assert first[0] == 0 and first[1] >= 3, first  # rows of both captures, the gather
assert run(1)[::2] == (0, 1) and run(1) == (0, 0, 1)
if wide:
    assert lib.fbp_batch_set_config(batch, 2, stream) == {unsupported}
    assert run(1) == (0, 0, 1)  # the captured graph
    assert run(0) == first
else:
    for nth in range(1, {allocations} + 1):
        _lib.check(lib.fbp_batch_set_config(batch, 0, stream))
        assert run(1)[::2] == (0, 1)
        fake.fake_fail_allocation(nth)
        st = lib.fbp_batch_set_config(batch, {config}, stream)
        fake.fake_fail_allocation(0)
        assert st == {oom}, st
        assert run(0) == ({oom}, 0, 0) and run(1) == ({oom}, 0, 0)
    _lib.check(lib.fbp_batch_set_config(batch, {config}, stream))
    assert run(0)[0] == 0 and run(1)[::2] == (0, 1)
    _lib.check(lib.fbp_batch_set_config(batch, 0, stream))
    assert run(0) == first
_lib.check(lib.fbp_batch_destroy(batch))
_lib.check(lib.fbp_destroy(ctx))
assert fake.fake_live_allocations() == 0
print("ok")
"""


@pytest.fixture(scope="module")
def fake(built, tmp_path_factory):
    so = tmp_path_factory.mktemp("fake") / "libfake_cudart.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", "/usr/local/cuda/include",
                    str(ROOT / "tests" / "cpp" / "fake_cudart.cpp"), "-o", str(so)], check=True)
    return so


def _run(fake, **kw):
    src = SCRIPT.format(root=str(ROOT), oom=2, unsupported=5, **kw)
    p = subprocess.run([sys.executable, "-c", src], env={**os.environ, "LD_PRELOAD": str(fake)}, capture_output=True,
                       text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout + p.stderr


def test_a_configuration_that_does_not_fit(fake):
    _run(fake, wide=True, allocations=0, config=2)


# Configuration 2 needs longer rows, 3 more work items.
@pytest.mark.parametrize("config,allocations", [(2, 1), (3, 1)])
def test_buffers_that_cannot_be_had(fake, config, allocations):
    _run(fake, wide=False, allocations=allocations, config=config)

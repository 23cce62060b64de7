"""The library's host code on a stand-in for the CUDA runtime (fake_cudart.cpp), each
test in a process of its own: what launches ask for and what failed calls leave
behind.  No GPU."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PRELUDE = f"""
import ctypes, importlib.util
spec = importlib.util.spec_from_file_location("wos_lib", r"{ROOT}/diff-wos_b200/wos/_lib.py")
_lib = importlib.util.module_from_spec(spec)
spec.loader.exec_module(_lib)
fake = ctypes.CDLL("libcudart.so.12")
fake.fake_live.restype = fake.fake_calls.restype = ctypes.c_longlong
fake.fake_fail_at.argtypes = [ctypes.c_longlong]
L = _lib.lib()
D = ctypes.c_void_p(1 << 30)  # a device address; nothing reads it
def create(dim, nV, nF):
    h = ctypes.c_void_p()
    rc = L.wos_scene_create(dim, D, nV, D, nF, D, 0, None, None, ctypes.byref(h))
    return rc, h
params = _lib.WosParams(4, 32, 1e-3, 0, 0, 0, 0, 0, 1, 0, 0)
adjoint = _lib.WosAdjointParams(1e-3, 0.1, 1, 1, 1e-3, 1, 1, 0)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("cudart")
    (d / "map").write_text("libcudart.so.12 { global: *; };\n")
    include = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", f"-I{include}", "-Wl,-soname,libcudart.so.12",
                    f"-Wl,--version-script={d / 'map'}", "-o", str(d / "libcudart.so.12"),
                    str(ROOT / "tests" / "fake_cudart.cpp")], check=True)

    def run(code):
        env = dict(os.environ, LD_LIBRARY_PATH=f"{d}:{os.environ.get('LD_LIBRARY_PATH', '')}")
        r = subprocess.run([sys.executable, "-c", PRELUDE + code], env=env, capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


def test_shared_memory_limits_are_never_lowered(fake):
    """A kernel's limit belongs to the process: a call for a shallow scene must not
    take away what another thread's call for a deep one is about to launch with."""
    fake("""
rc, deep = create(3, 100000, 81920)
assert rc == 0
rc, shallow = create(3, 100, 80)
assert rc == 0
for scene in (deep, shallow, deep):
    for call in (
        lambda: L.wos_solve(scene, D, 10, ctypes.byref(params), D, D, None, 0, None),
        lambda: L.wos_solve_adjoint(scene, D, 10, ctypes.byref(params), ctypes.byref(adjoint), 1, None, D, None, D,
                                    D, D, None, None, 0, None),
        lambda: L.wos_adjoint(scene, D, 10, ctypes.byref(params), ctypes.byref(adjoint), D, D, D, None, None, 0, None),
        lambda: L.wos_soft_walk(scene, D, 10, ctypes.byref(params), None, None, D, D, None, None, None, 0, None),
        lambda: L.wos_soft_walk_adjoint(scene, D, 10, ctypes.byref(params), D, D, D, None),
    ):
        rc = call()
        assert rc == 0, L.wos_last_error_string()
    item = (_lib.WosBatchItem * 1)(_lib.WosBatchItem(scene.value, D.value, 10, 1, None, params))
    plan = ctypes.c_void_p()
    assert L.wos_batch_create(item, 1, ctypes.byref(adjoint), 1, None, ctypes.byref(plan)) == 0
    assert L.wos_batch_run(plan, 0, None) == 0
    assert L.wos_batch_destroy(plan, None) == 0
assert fake.fake_launches() > 0 and fake.fake_refused() == 0
assert fake.fake_lowered() == 0, fake.fake_lowered()
""")


@pytest.mark.parametrize("nF", [134217728, 134217729, 300000000])
def test_meshes_above_65536_split_segments_are_taken(fake, nF):
    """Segments of 2,048 triangles and the coordinate within them share a sort key."""
    fake(f"""
rc, h = create(3, 1000000, {nF})
assert rc == 0, L.wos_last_error_string()
assert L.wos_scene_update_vertices(h, D, None) == 0
L.wos_scene_destroy(h, None)
assert fake.fake_live() == 0
""")


@pytest.mark.parametrize("dim,nV,nF", [(2, 500, 500), (3, 50, 1), (3, 3000, 5000)])
def test_failed_builds_leave_nothing_allocated(fake, dim, nV, nF):
    """Every call of a scene's making and of a rebuild fails once."""
    fake(f"""
fake.fake_fail_at(0)
rc, scene = create({dim}, {nV}, {nF})
assert rc == 0
made, held = fake.fake_calls(), fake.fake_live()
fake.fake_fail_at(0)
assert L.wos_scene_update_vertices(scene, D, None) == 0
moved = fake.fake_calls()
assert fake.fake_live() == held
for k in range(1, moved + 1):
    fake.fake_fail_at(k)
    assert L.wos_scene_update_vertices(scene, D, None) == _lib.WOS_ERR_CUDA, k
    assert fake.fake_live() == held, k
for k in range(1, made + 1):
    fake.fake_fail_at(k)
    rc, h = create({dim}, {nV}, {nF})
    assert rc == _lib.WOS_ERR_CUDA and not h.value, k
    assert fake.fake_live() == held, k
""")


@pytest.mark.parametrize("sample", [1.0, 0.001])
def test_slot_tuner_times_the_launches_of_a_step(fake, sample):
    """One launch per phase over the items of every depth, and the chunk that the step
    would grab with the candidate."""
    fake(f"""
scenes = [create(3, 1000, nF)[1] for nF in (80, 5000, 80000)]
big = _lib.WosParams(256, 32, 1e-3, 0, 0, 0, 0, 0, 1, 0, 0)
item = (_lib.WosBatchItem * 3)(*[_lib.WosBatchItem(h.value, D.value, 100000, 1, None, big) for h in scenes])
plan = ctypes.c_void_p()
assert L.wos_batch_create(item, 3, ctypes.byref(adjoint), 1, None, ctypes.byref(plan)) == 0
held = fake.fake_live()
shapes = [(256, 0, 16), (256, 0, 64), (256, 0, 128), (512, 2, 128)]
arr = [(ctypes.c_int32 * 4)(*v) for v in zip(*shapes)]
for kernel, arg, slot in (("k_walk_batch", 7, (3, 0)), ("k_adjoint_batch", 9, (3, 1))):
    step = []
    for s in shapes:
        assert L.wos_batch_set_launch_slot(plan, *slot, *s) == 0
        fake.fake_watch(kernel.encode(), arg)
        assert L.wos_batch_run(plan, 0, None) == 0
        assert fake.fake_seen(1) == -1
        step.append(fake.fake_seen(0))
    assert len(set(step)) > 2
    fake.fake_watch(kernel.encode(), arg)
    assert L.wos_batch_autotune_slots(plan, *arr, 4, 1, {sample}, None, None, None) == 0
    tuned = [fake.fake_seen(i) for i in range(1, 6)]  # after the full step's
    assert tuned == step + [-1], (tuned, step)
assert fake.fake_live() == held
""")

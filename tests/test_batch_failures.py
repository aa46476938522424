"""A batch that fails half-way: what was launched before is waited for by the caller's stream, and nothing is
launched before every scene's state is in place.  The host code runs on a fake CUDA runtime
(fake_cuda.cpp) whose allocations and launches fail on request, in a process of its own."""
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

import pytest

from sharpray_gb300.build import CSRC, HOST_SOURCES, ROOT, cuda_home

CHILD = """
import ctypes as C, sys
from sharpray_gb300 import Context, SharpRayError, _abi, render_batch, render_params, synth
lib = _abi.load(sys.argv[1])
lib.fake_log.restype = C.c_char_p
ctx = Context(0)
descs = [synth.config_c1(40 + 8 * i, 24, 2) for i in range(3)]
scenes = [d.instantiate(ctx) for d in descs]
for s in scenes:
    s.build()
aovs = [_abi.SrAovs(*[1] * 7) for _ in descs]
def batch():
    try:
        render_batch(scenes, [d.view for d in descs], [render_params(*d.render_args()) for d in descs], aovs, 99)
        return "ok"
    except SharpRayError as e:
        return str(e.code)
lib.fake_reset(int(sys.argv[2]), int(sys.argv[3]))
print(batch())
print(lib.fake_log().decode())
lib.fake_reset(0, 0)
print("again " + batch())
"""


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake_cuda")
    inc = [f"-I{ROOT / 'include'}", f"-I{CSRC}", f"-I{cuda_home() / 'include'}"]
    sources = [CSRC / s for s in HOST_SOURCES] + [ROOT / "tests" / "fake_cuda.cpp"]

    def compile_one(src):
        obj = out / (src.name + ".o")
        subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", *inc, "-c", str(src), "-o", str(obj)], check=True)
        return str(obj)

    with ThreadPoolExecutor() as ex:
        objects = list(ex.map(compile_one, sources))
    lib = out / "libfake.so"
    subprocess.run(["g++", "-shared", *objects, "-o", str(lib)], check=True)
    return lib


def run(lib, malloc_to_fail, launch_to_fail):
    r = subprocess.run([sys.executable, "-c", CHILD, str(lib), str(malloc_to_fail), str(launch_to_fail)], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    lines = r.stdout.split("\n")
    assert lines[-2] == "again ok"
    return lines[0], [line.split() for line in lines[1:-2] if line]


def joined(log):
    """Every launch on another stream than the caller's (99) is followed by an event there that the caller's
    stream waits for, or by a wait of the host."""
    for i, op in enumerate(log):
        if op[0] != "launch" or op[1] == "99":
            continue
        events = {o[2]: j for j, o in enumerate(log) if j > i and o[:2] == ["record", op[1]]}
        waits = [j for j, o in enumerate(log) if o[:2] == ["wait", "99"] and o[2] in events and j > events[o[2]]]
        syncs = [j for j, o in enumerate(log) if j > i and (o == ["sync", op[1]] or o == ["sync", "device"])]
        if not waits and not syncs:
            return False
    return True


def launches(log):
    return [op for op in log if op[0] == "launch"]


def test_whole_batch(fake_lib):
    said, log = run(fake_lib, 0, 0)
    assert said == "ok" and len(launches(log)) == 3 and joined(log)
    allocations = [i for i, op in enumerate(log) if op == ["malloc"]]
    assert allocations and max(allocations) < log.index(launches(log)[0]), "state is allocated before the first launch"


# the path state of the first, second and third scene (an allocation each)
@pytest.mark.parametrize("nth", [1, 2, 3])
def test_allocation_fails(fake_lib, nth):
    said, log = run(fake_lib, nth, 0)
    assert said != "ok" and not launches(log)


@pytest.mark.parametrize("nth", [1, 2, 3])
def test_launch_fails(fake_lib, nth):
    said, log = run(fake_lib, 0, nth)
    assert said != "ok" and len(launches(log)) == nth and joined(log)

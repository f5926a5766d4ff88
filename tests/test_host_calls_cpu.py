"""Host-buffer calls and the memory they work on, without a device: the library's
C++ objects linked with a stand-in of the CUDA runtime (host_calls_fake.cpp).

* A host call begun while another of the same context is in flight (as a second
  thread does) leaves the other's memory alone.
* A call that fails half-way returns its error with nothing of its work in flight.
* A call that succeeds does so too: a scene can be used on any stream at once.
* What calls keep for the next one is bounded and goes back with tpt_context_trim.
* A scene without materials, which nothing can shade, holds no shading records.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "toy-path-tracing_b200")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    names = [os.path.join(d, f[:-4]) for d in ("api", "host")
             for f in sorted(os.listdir(os.path.join(PKG, "csrc", d))) if f.endswith(".cpp")]
    objects = ["_build/obj/%s.o" % n for n in names]
    subprocess.run(["make", "-s", "-j4", "-C", PKG] + objects, check=True)
    exe = str(tmp_path_factory.mktemp("host_calls") / "host_calls_fake")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    # kernels that no call here launches stay unresolved
    subprocess.run(["g++", "-std=c++17", "-O1", "-no-pie", "-I", os.path.join(cuda, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "host_calls_fake.cpp")] + [os.path.join(PKG, o) for o in objects]
                   + ["-lpthread", "-Wl,--unresolved-symbols=ignore-all"], check=True)
    return exe


def run(program, *args):
    r = subprocess.run([program, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", (args, r.returncode, r.stdout, r.stderr)


@pytest.mark.parametrize("outer,inner", [
    ("traverse_pinned", "render"), ("traverse_pinned", "render_large"), ("traverse_pinned", "upload"),
    ("traverse_pageable", "render_batch"), ("traverse_pageable", "upload_large"),
    ("render", "upload"), ("render", "upload_large"), ("render_batch", "upload"),
])
def test_calls_in_flight_keep_their_memory(program, outer, inner):
    run(program, "share", outer, inner)


# three or more launches: a query of 300,001 rays in chunks, one traversal per bounce
# and the image of a render, three jobs of a batch
@pytest.mark.parametrize("call", ["traverse_pinned", "traverse_pageable", "render", "render_own_memory", "render_batch"])
@pytest.mark.parametrize("launch", [1, 2, 3])
def test_failed_calls_leave_nothing_in_flight(program, call, launch):
    run(program, "fail", call, str(launch))


@pytest.mark.parametrize("call", ["upload", "upload_large", "traverse_pinned", "traverse_pageable", "render",
                                  "render_own_memory", "render_batch"])
def test_calls_leave_nothing_in_flight(program, call):
    run(program, "wait", call, "1")


@pytest.mark.parametrize("triangles", [100, 5000])
def test_scenes_for_queries_hold_no_shading_records(program, triangles):
    run(program, "records", str(triangles), "96")


# a query of 300,001 rays: 7 + 2 planes on the device, 9 planes of two chunks in staging
@pytest.mark.parametrize("call,mib", [("upload", 128), ("upload_large", 128), ("render", 128), ("render_large", 128),
                                      ("render_batch", 128), ("traverse_pinned", 11), ("traverse_pageable", 16)])
def test_kept_memory_is_bounded_and_given_back(program, call, mib):
    run(program, "trim", call, str(mib))

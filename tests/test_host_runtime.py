"""The library's host code against a CUDA runtime without a GPU (fake_cudart.c, preloaded):
what it allocates, clears and launches, on which stream, and what it does when memory runs
out.  No kernel runs."""
import json
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

PRELUDE = """
import ctypes, json, re, sys
import numpy as np
import lux_b200 as L

fake = ctypes.CDLL(None)
fake.fake_log.restype = ctypes.c_char_p
fake.fake_used.restype = ctypes.c_size_t
fake.fake_set_limit.argtypes = [ctypes.c_size_t]


def log(clear=True):
    text = fake.fake_log().decode()
    if clear:
        fake.fake_clear_log()
    return text.splitlines()


def launched(lines):
    # Kernel names of the launches: the k_... part of the mangled name.
    return [re.search(r"(k_[a-z_]*[a-z])", s).group(1) for s in lines if s.startswith("launch")]


def triangles(n, seed=0):
    return np.random.default_rng(seed).random((n, 9), np.float32)


ctx = L.Context(0)
"""


@pytest.fixture(scope="session")
def run(tmp_path_factory):
    """run(code): code's result (its variable `out`) in a process with the fake runtime."""
    lib = tmp_path_factory.mktemp("fake") / "fake_cudart.so"
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", str(lib),
                    os.path.join(HERE, "fake_cudart.c"), "-lpthread"], check=True)

    def call(code):
        env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=ROOT)
        res = subprocess.run([sys.executable, "-c", PRELUDE + code + "\nprint(json.dumps(out))"],
                             env=env, capture_output=True, text=True, timeout=120)
        assert res.returncode == 0, res.stderr
        return json.loads(res.stdout.splitlines()[-1])

    return call


def test_a_new_bvh_is_cleared_in_stream_order(run):
    """What a build relies on finding cleared is cleared on the context's stream: a memset on
    the default stream has no order with a build on a non-blocking one."""
    lines = run("""
log()
bvh = ctx.build_lbvh(triangles(5000))
out = log()
""")
    memsets = [s for s in lines if s.startswith("memset")]
    assert len(memsets) >= 2 and not any("default" in s for s in memsets), memsets


def test_the_error_word_is_cleared_in_stream_order(run):
    """The context's words and a reported error word are cleared on the context's stream: a
    clear on the default stream can land after the next call's kernels and lose their errors."""
    out = run("""
start = log()
word = ctypes.c_int.from_address(int(re.match(r"malloc 4 (0x[0-9a-f]+)", next(
    s for s in start if s.startswith("malloc 4 "))).group(1), 16))
word.value = 4
try:
    ctx.synchronize()
    status = 0
except L.LuxError as e:
    status = e.status
ctx.synchronize()
out = [start + log(), status, word.value]
""")
    memsets = [s for s in out[0] if s.startswith("memset")]
    assert out[1] == 5 and out[2] == 0
    assert len(memsets) == 3 and not any("default" in s for s in memsets), memsets


def test_a_rebuild_that_found_no_memory_leaves_an_empty_bvh(run):
    """After a rebuild that was refused its memory the BVH holds nothing: the next smaller
    rebuild allocates anew instead of launching on arrays that are gone."""
    out = run("""
bvh = ctx.build_lbvh(triangles(1000))
fake.fake_set_limit(fake.fake_used() + (1 << 20))
log()
try:
    bvh.rebuild(triangles(100000))
    status = 0
except L.LuxError as e:
    status = e.status
refused = log()
bvh.rebuild(triangles(2000))
out = [status, refused, log()]
""")
    status, refused, again = out
    assert status == 3 and not any(s.startswith("launch") for s in refused)
    first_launch = next(i for i, s in enumerate(again) if s.startswith("launch"))
    sizes = [int(s.split()[1]) for s in again[:first_launch] if s.startswith("malloc")]
    assert max(sizes, default=0) > 100 * 2000, again


def test_a_build_needs_no_room_for_the_wide_nodes(run):
    """Where a triangle BVH's 4-wide nodes do not fit beside its other arrays, the build still
    succeeds, as it does for a BVH that is only refitted or downloaded; the first ray query asks
    for them again."""
    out = run("""
n = 200000
bvh = ctx.build_lbvh(triangles(n))           # grows the context's scratch and staging
bvh.close()
rays = np.zeros((64, 8), np.float32)
used = fake.fake_used()
log()
fake.fake_set_limit(used + 160 * n)
bvh = ctx.build_lbvh(triangles(n))
bvh.refit(triangles(n))
built = log()
try:
    bvh.trace_closest(rays)
    status = 0
except L.LuxError as e:
    status = e.status
fake.fake_set_limit(used + 400 * n)
bvh.trace_closest(rays)
bvh.close()
out = [status, launched(built), fake.fake_used() - used, log()]
""")
    status, kernels, left, rest = out
    assert "k_climb" in kernels and status == 3
    assert left == 0 and not any("unknown" in s for s in rest)


def test_a_server_accounts_for_the_pools_it_allocates(run):
    """bytes_in_use of an idle server is what its path pools took, and none of their arrays is
    a per-path array that only single renders use."""
    out = run("""
from lux_b200 import scene as S, server as SV
scene = S.Scene(ctx, S.make_cornell_scene(32, 32))
out = []
for paths in (1 << 14, 1 << 15):
    log()
    with SV.Server([scene], pool_paths=paths) as srv:
        out.append([srv.stats()["bytes_in_use"],
                    [int(s.split()[1]) for s in log() if s.startswith("malloc")]])
""")
    (small, a), (large, b) = out
    per_path = [y - x for x, y in zip(a, b)]         # what grows with the pool
    assert large - small == sum(per_path) and small == sum(per_path), (small, sum(per_path))
    # state, ray, radiance and request of two pools; shadow, hit, shadow queue, where a shadow
    # ray's path went, ended paths
    assert small == (1 << 14) * (2 * (64 + 32 + 16 + 4) + 64 + 16 + 4 + 4 + 4)


def test_a_mesh_update_uploads_in_stream_order(run):
    """Everything a mesh's first update uploads goes through the context's stream, on which its
    kernels read it: a pageable copy on the default stream may still be on its way when they
    start."""
    lines = run("""
from lux_b200 import scene as S
scene = S.Scene(ctx, S.make_cornell_scene(32, 32))
log()
scene.update_mesh(0, np.zeros((36, 3), np.float32))
out = log()
""")
    copies = [s for s in lines if s.startswith("memcpy")]
    assert len(copies) >= 3 and not any("default" in s for s in copies), copies


def test_the_first_refit_after_a_build_is_one_launch(run):
    """The build leaves all that a refit reads: no pass of its own over the nodes."""
    out = run("""
out = []
for n in (1000, 5000, 20000):
    bvh = ctx.build_lbvh(triangles(n))
    for again in range(2):
        log()
        bvh.refit(triangles(n, 1))
        out.append(launched(log()))
""")
    assert out == [["k_refit"]] * 6, out


def test_the_autotuner_tries_every_smaller_grid(run):
    """Resident blocks per SM below those that fit: three fit batches of up to 2^20 paths, four
    larger ones."""
    out = run("""
from lux_b200 import autotune as A, scene as S
scene = S.Scene(ctx, S.make_cornell_scene(32, 32))
out = []
for spp in (4, 2048):
    log()
    A.autotune_render(ctx, scene, S.request(32, 32, spp, 0))
    sm = 148
    grids = [int(s.split(" grid ")[1].split()[0]) for s in log() if "k_walk" in s]
    out.append(sorted({g // sm for g in grids}))
""")
    assert out == [[1, 2, 4], [1, 2, 3, 4]], out    # (the stand-in says that four blocks fit)


def test_the_film_encoder_leaves_the_builds_scratch_alone(run):
    """Host films go through the context's staging, which every call that uses it waits for:
    a build may still be sorting in the scratch on a stream that the context had before."""
    out = run("""
film, ppm = np.ones((40, 30, 3), np.float32), np.zeros((40, 30, 3), np.uint8)
log()
lib = ctx._lib
L._check(lib.lux_film_encode(ctx.handle, film.ctypes.data, 30, 40, 1, 0, ppm.ctypes.data))
out = [ctx.get_option(L.OPT_SCRATCH_BYTES), ctx.get_option(L.OPT_STAGING_BYTES), launched(log())]
""")
    assert out[0] == 0 and out[1] >= 40 * 30 * 15 and out[2] == ["k_encode"], out

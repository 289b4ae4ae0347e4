"""The GPU LBVH build (rt_build_bvh_device) must emit exactly the node array
of the oracle's transcription of the six S1 passes (ModelSpaceToWorldSpace.comp
to ConstructAABBsOfInternalNodes.comp), and of the host build."""
import itertools
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent


def run_child(script):
    """The script in a process of its own (argv: the repository's root)."""
    r = subprocess.run([sys.executable, "-c", script, str(ROOT)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]


def device_build(rt, torch, tris, spheres=None, mode=0):
    tris = np.ascontiguousarray(tris, dtype=rt.TRIANGLE_DTYPE)
    n = len(tris) + (0 if spheres is None else len(spheres))
    d_t = torch.from_numpy(tris.view(np.uint8)).cuda() if len(tris) else None
    d_s = None if spheres is None else torch.from_numpy(np.ascontiguousarray(spheres).view(np.uint8)).cuda()
    d_n = torch.full((max(2 * n - 1, 1) * 40,), 0xCC, dtype=torch.uint8, device="cuda")
    rt.build_bvh_device(d_t, len(tris), d_s, 0 if spheres is None else len(spheres), d_n, bvh_mode=mode)
    torch.cuda.synchronize()
    return d_n.cpu().numpy().view(rt.NODE_DTYPE)[: 2 * n - 1]


@pytest.mark.parametrize("mode", [0, 1])
def test_device_build_matches_host(rt, cuda, mode):
    tris, _, _ = rt.gen_config1()
    assert np.array_equal(device_build(rt, cuda, tris, mode=mode).view(np.uint8),
                          rt.build_bvh(tris, bvh_mode=mode).view(np.uint8))
    soup = rt.gen_soup(6, 0, 300_000, 1.0, 0.002)
    sph = np.zeros(13, rt.SPHERE_DTYPE)
    sph["center"][:, :3] = np.random.default_rng(3).random((13, 3)).astype(np.float32)
    sph["radius"] = np.float32(0.02)
    assert np.array_equal(device_build(rt, cuda, soup, sph, mode).view(np.uint8),
                          rt.build_bvh(soup, sph, bvh_mode=mode).view(np.uint8))


def test_device_build_edge_cases(rt, cuda):
    t = rt.gen_soup(3, 5, 70_000, 1.0, 0.01)
    for n in (1, 2, 3, 255, 4096, 4097, 65_537):
        for mode in (0, 1):
            assert np.array_equal(device_build(rt, cuda, t[:n], mode=mode).view(np.uint8),
                                  rt.build_bvh(t[:n], bvh_mode=mode).view(np.uint8)), n
    same = np.repeat(t[:1], 5000)  # equal codes everywhere: index tie-break
    assert np.array_equal(device_build(rt, cuda, same).view(np.uint8), rt.build_bvh(same).view(np.uint8))


def test_device_build_config3_and_scene(rt, cuda):
    tris = rt.gen_soup(3, 0, 4_194_304, 1.0, 0.002)
    host = rt.build_bvh(tris)
    assert np.array_equal(device_build(rt, cuda, tris).view(np.uint8), host.view(np.uint8))
    with rt.Scene(tris[:200_000], build_on_device=True) as a, rt.Scene(tris[:200_000]) as b:
        assert np.array_equal(a.nodes().view(np.uint8), b.nodes().view(np.uint8))


@pytest.mark.parametrize("mode", [0, 1], ids=["sorted", "reference"])
def test_device_build_matches_oracle(rt, orc, cuda, mode):
    """The device build against the oracle's transcription of the S1 passes
    (which the CPU suite pins to the reference's own shaders in reference
    mode): config 1, a soup with spheres, duplicate centroids, the full
    config-3 soup, and sizes around the device kernels' block sizes."""
    tris, _, _ = rt.gen_config1()
    assert np.array_equal(device_build(rt, cuda, tris, mode=mode).view(np.uint8),
                          orc.build_bvh(tris, mode=mode)[0].view(np.uint8))
    soup = rt.gen_soup(8, 0, 200_000, 1.0, 0.002)
    sph = np.zeros(40, rt.SPHERE_DTYPE)
    sph["center"][:, :3] = np.random.default_rng(8).random((40, 3)).astype(np.float32)
    sph["radius"] = np.float32(0.01)
    assert np.array_equal(device_build(rt, cuda, soup, sph, mode).view(np.uint8),
                          orc.build_bvh(soup, spheres=sph, mode=mode)[0].view(np.uint8))
    dup = np.concatenate([soup[:500]] * 6)
    assert np.array_equal(device_build(rt, cuda, dup, mode=mode).view(np.uint8),
                          orc.build_bvh(dup, mode=mode)[0].view(np.uint8))
    for n in (1, 2, 255, 256, 257, 1023, 1025):
        assert np.array_equal(device_build(rt, cuda, soup[:n], mode=mode).view(np.uint8),
                              orc.build_bvh(soup[:n], mode=mode)[0].view(np.uint8)), n
    big = rt.gen_soup(3, 0, 4_194_304, 1.0, 0.002)
    assert np.array_equal(device_build(rt, cuda, big, mode=mode).view(np.uint8),
                          orc.build_bvh(big, mode=mode)[0].view(np.uint8))


@pytest.mark.parametrize("n", [1024, 1025, 1_048_576, 1_048_577, 1_052_673, 3_145_728, 3_145_729])
def test_device_build_sort_tiles(rt, cuda, n):
    """Sizes at the edges of the radix sort's tiles and where its tile size changes, for scattered codes and
    for a few long runs of equal ones."""
    soup = rt.gen_soup(9, 0, n, 1.0, 0.004)
    assert np.array_equal(device_build(rt, cuda, soup).view(np.uint8), rt.build_bvh(soup).view(np.uint8))
    runs = soup[np.arange(n) * 7 // n]
    assert np.array_equal(device_build(rt, cuda, runs).view(np.uint8), rt.build_bvh(runs).view(np.uint8))


@pytest.mark.parametrize("n", [511, 512, 513, 1024, 1537, 40_961, 65_536, 65_537, 131_073, 300_001])
@pytest.mark.parametrize("shape", ["soup", "equal", "line"])
def test_device_build_tree_blocks(rt, cuda, n, shape):
    """Sizes at the edges of the tree kernel's blocks: shallow trees, one code everywhere (the index decides)
    and a line of clusters (long ranges over many blocks); arrays that are only 4-byte aligned too."""
    t = rt.gen_soup(11, 0, n, 1.0, 0.01)
    if shape == "equal":
        t = np.repeat(t[:1], n)
    elif shape == "line":
        for v in ("v0", "v1", "v2"):
            t[v][:, 0] += (2.0 ** (np.arange(n) % 23)).astype(np.float32)
    want = rt.build_bvh(t).view(np.uint8)
    assert np.array_equal(device_build(rt, cuda, t).view(np.uint8), want)
    raw = cuda.zeros(n * 64 + 4, dtype=cuda.uint8, device="cuda")
    raw[4:] = cuda.from_numpy(t.view(np.uint8)).cuda()
    out = cuda.zeros((2 * n - 1) * 40 + 4, dtype=cuda.uint8, device="cuda")
    rt.build_bvh_device(raw[4:], n, d_nodes=out[4:])
    assert np.array_equal(out[4:].cpu().numpy(), want)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 8_191, 8_193, 16_383, 16_384, 16_385])
def test_device_build_cluster_sizes(rt, cuda, n):
    """Sizes at the edges of the one-cluster front (blocks without keys, the last size that fits) in both modes,
    with equal codes and with spheres among the primitives."""
    t = rt.gen_soup(12, 0, n, 1.0, 0.01)
    for mode in (0, 1):
        assert np.array_equal(device_build(rt, cuda, t, mode=mode).view(np.uint8),
                              rt.build_bvh(t, bvh_mode=mode).view(np.uint8)), mode
    few = t[np.arange(n) * 3 // n]
    assert np.array_equal(device_build(rt, cuda, few).view(np.uint8), rt.build_bvh(few).view(np.uint8))
    sph = np.zeros(min(n, 50), rt.SPHERE_DTYPE)
    sph["center"][:, :3] = np.random.default_rng(12).random((len(sph), 3)).astype(np.float32)
    sph["radius"] = np.float32(0.02)
    part = t[: n - len(sph)]
    assert np.array_equal(device_build(rt, cuda, part, sph).view(np.uint8), rt.build_bvh(part, sph).view(np.uint8))


def test_device_build_scratch_is_given_back(rt, cuda):
    """Builds on two streams at once and back to back with a synchronisation between them are right; what the
    library keeps between builds is bounded and goes back with rt_stream_release."""
    t = [rt.gen_soup(13, k, 300_000 + 50_001 * k, 1.0, 0.004) for k in range(2)]
    want = [rt.build_bvh(x).view(np.uint8) for x in t]
    d_t = [cuda.from_numpy(x.view(np.uint8)).cuda() for x in t]
    d_n = [cuda.zeros((2 * len(x) - 1) * 40, dtype=cuda.uint8, device="cuda") for x in t]
    streams = [cuda.cuda.Stream() for _ in t]
    cuda.cuda.synchronize()
    for _ in range(3):
        for k in range(2):
            rt.build_bvh_device(d_t[k], len(t[k]), d_nodes=d_n[k], stream=streams[k])
    cuda.cuda.synchronize()
    for k in range(2):
        assert np.array_equal(d_n[k].cpu().numpy(), want[k])
    rt.release_stream()
    free0 = cuda.cuda.mem_get_info()[0]
    rt.build_bvh_device(d_t[0], len(t[0]), d_nodes=d_n[0])
    cuda.cuda.synchronize()
    assert free0 - cuda.cuda.mem_get_info()[0] <= 256 << 20
    rt.release_stream()
    assert free0 - cuda.cuda.mem_get_info()[0] <= 4 << 20
    assert np.array_equal(d_n[0].cpu().numpy(), want[0])


@pytest.mark.parametrize("part", ["all", "one_group"])
def test_device_build_long_lists(rt, cuda, part):
    """Codes with at most five bits set: deep one-sided subtrees everywhere, so that a group of blocks leaves more
    nodes for the top of the tree than one block takes (1,850 of 174,438 primitives' middle group, 1,870 of
    65,536 primitives in one group; the limit is 1,792)."""
    codes = np.array(sorted([0] + [sum(1 << b for b in c) for k in range(1, 6)
                                   for c in itertools.combinations(range(30), k)]), np.int64)
    q = np.zeros((len(codes), 3))
    for b in range(30):
        q[:, b % 3] += ((codes >> b) & 1) * (1 << (b // 3))
    if part == "one_group":
        q = np.concatenate([q[:1], q[70_000:70_000 + 65_534]])
    centre = np.concatenate([(q + 0.5) / 1024, [[1.0 - 0.4 / 1024] * 3]]).astype(np.float32)
    t = np.zeros(len(centre), rt.TRIANGLE_DTYPE)
    for v, d in (("v0", (-1, 0, 0)), ("v1", (0.5, 1, 0)), ("v2", (0.5, -1, 0))):
        t[v][:, :3] = centre + np.float32(1e-5) * np.array(d, np.float32)
    assert np.array_equal(device_build(rt, cuda, t).view(np.uint8), rt.build_bvh(t).view(np.uint8))


@pytest.mark.parametrize("traced", [False, True], ids=["builds_only", "with_a_workspace"])
def test_release_waits_for_the_build(rt, cuda, traced):
    """rt_stream_release straight after a build, which is still running: its scratch (86 MB) goes back too, also on
    a stream that has no workspace."""
    tris = rt.gen_soup(14, 0, 4_194_304, 1.0, 0.002)
    d_t = cuda.from_numpy(tris.view(np.uint8)).cuda()
    d_n = cuda.zeros((2 * len(tris) - 1) * 40, dtype=cuda.uint8, device="cuda")
    rays = cuda.zeros(32, dtype=cuda.uint8, device="cuda")
    hits = cuda.zeros(8, dtype=cuda.uint8, device="cuda")
    stream = cuda.cuda.Stream()
    with rt.Scene(tris[:100]) as sc:
        for turn in range(2):
            cuda.cuda.synchronize()
            if traced:
                sc.trace(rays, hits, n=1, stream=stream)
            rt.build_bvh_device(d_t, len(tris), d_nodes=d_n, stream=stream)
            rt.release_stream(stream)
            cuda.cuda.synchronize()
            if turn == 0:  # whatever is kept from builds before this test
                rt.release_stream()
                free = cuda.cuda.mem_get_info()[0]
    assert free - cuda.cuda.mem_get_info()[0] <= 4 << 20
    assert np.array_equal(d_n.cpu().numpy(), rt.build_bvh(tris).view(np.uint8).ravel())


RESET = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import raytracergpu_mastersproject_gb300 as rt
L, runtime = rt.lib(), C.CDLL("/usr/local/cuda/lib64/libcudart.so")
L.rt_device_alloc.argtypes = [C.c_size_t, C.POINTER(C.c_void_p)]
L.rt_copy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p]
tris = rt.gen_soup(3, 0, 5000, 1.0, 0.01)
want = rt.build_bvh(tris).view(np.uint8).ravel()
for turn in range(3):
    d_t, d_n = C.c_void_p(), C.c_void_p()
    assert L.rt_device_alloc(tris.nbytes, C.byref(d_t)) == 0 and L.rt_device_alloc(want.nbytes, C.byref(d_n)) == 0
    assert L.rt_copy(d_t.value, tris.ctypes.data, tris.nbytes, None) == 0
    assert L.rt_build_bvh_device(d_t.value, len(tris), None, 0, 0, d_n.value, None) == 0, L.rt_last_error_string()
    got = np.zeros_like(want)
    assert L.rt_copy(got.ctypes.data, d_n.value, got.nbytes, None) == 0 and L.rt_stream_wait(None, 10.0) == 0
    assert np.array_equal(got, want)
    if turn == 1:
        assert L.rt_stream_release(None) == 0
    assert runtime.cudaDeviceReset() == 0
assert L.rt_stream_release(None) == 0  # nothing of the present context to give back
"""


def test_device_build_after_a_device_reset(cuda):
    """The pool of the builds' scratch belongs to a context: a build after cudaDeviceReset takes a new one."""
    run_child(RESET)


CAPTURE = r"""
import sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
import raytracergpu_mastersproject_gb300 as rt
for n in (5_000, 20_482, 300_000):  # one cluster, one group of tree blocks, several
    soups = [rt.gen_soup(20 + k, 0, n, 1.0, 0.01) for k in range(2)]
    want = [rt.build_bvh(t).view(np.uint8).ravel() for t in soups]
    d_s = [torch.from_numpy(t.view(np.uint8)).cuda() for t in soups]
    d_t, d_n = d_s[0].clone(), torch.zeros((2 * n - 1) * 40, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rt.build_bvh_device(d_t, n, d_nodes=d_n, stream=torch.cuda.current_stream())
    for k in (0, 1, 0):
        d_t.copy_(d_s[k])
        d_n.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(d_n.cpu().numpy(), want[k]), (n, k)
"""


def test_device_build_in_a_captured_graph(cuda):
    """A captured build, the process's first one among them, replays on what the triangles are by then."""
    run_child(CAPTURE)

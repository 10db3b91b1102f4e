"""Which path a precision-32 run takes and that both give the same bits, over
the sizes of the whole-run kernel: one block, clusters of every number of tiles
(padded to a power of two), grids up to a block an SM, and one tile more, which
goes by launches.  In a child process with launch_watch.c in front of the CUDA
runtime."""
import ctypes
import json
import os
import subprocess
import sys
import time

import numpy as np
import pytest

from conftest import ROOT, dev

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, json, sys
import numpy as np
import torch
import vsmc_gb300 as vc

watch = ctypes.CDLL(None)
watch.launch_watch_count.restype = ctypes.c_long
T = 12
rng = np.random.default_rng(3)
obs = np.cumsum(rng.normal(0, 0.3, (T, 2)), 0)


def run(n, scheme, graph, refuse=0, runs=1):
    pf = vc.ParticleFilter(n, 32, scheme, 0.5, seed=11, max_steps=T)
    pf.use_graph(graph)
    watch.launch_watch_refuse(refuse)
    counts = []
    for _ in range(runs):
        before = watch.launch_watch_count()
        h = pf.run(obs)
        counts.append(watch.launch_watch_count() - before)
    watch.launch_watch_refuse(0)
    s, w = pf.state_ptrs()
    ld = (n + 255) // 256 * 256

    class View:
        owner = pf
        __cuda_array_interface__ = {
            "data": (s, False), "shape": (4 * ld,), "strides": None,
            "typestr": "<i4", "version": 3}

    state = torch.as_tensor(View(), device="cuda").cpu().numpy()
    pf.close()
    return h, state.reshape(4, ld)[:, :n], counts


out = []
sms = torch.cuda.get_device_properties(0).multi_processor_count
for n, refuse in json.loads(sys.argv[1]):
    n = n if n > 0 else 1024 * sms - 1 - n
    for scheme in (vc.STRATIFIED, vc.SYSTEMATIC):
        a, sa, ca = run(n, scheme, True, refuse, 2)
        b, sb, cb = run(n, scheme, False)
        same = all(np.array_equal(a[k], b[k]) for k in a)
        out.append([n, refuse, ca, cb, bool(same and np.array_equal(sa, sb)),
                    int(a["resampled"].sum())])
print(json.dumps(out))
"""

# a block's tile is 1024 particles; 0, -1, -2: 1024 SMs - 1, + 0, + 1
SIZES = [2, 1000, 1024, 1025, 2048, 2049, 3073, 4097, 5121, 6145, 7169, 8192,
         8193, 20000, 100003, 0, -1, -2]


@pytest.fixture(scope="module")
def child(vc, tmp_path_factory):
    so = tmp_path_factory.mktemp("watch") / "watch.so"
    subprocess.check_call(
        ["gcc", "-O1", "-shared", "-fPIC", "-I/usr/local/cuda/include",
         os.path.join(ROOT, "tests", "cpp", "launch_watch.c"), "-o", str(so),
         "-ldl"])

    def go(cases):
        env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
        r = subprocess.run([sys.executable, "-c", CHILD, json.dumps(cases)],
                           capture_output=True, text=True, env=env, cwd=ROOT)
        assert r.returncode == 0, r.stderr[-3000:]
        return json.loads(r.stdout.splitlines()[-1])
    return go


def test_paths_and_bits(child):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n, _, graph, launches, same, resampled in child(
            [[n, 0] for n in SIZES]):
        assert graph == ([1, 1] if n <= 1024 * sms else [0, 0]), n
        assert launches == [0], n
        assert same, n
        assert resampled > 0 or n < 32, n


def test_a_refused_launch_goes_by_launches(child):
    """The runtime refuses cooperative launches (and this watch cluster ones):
    the run is the same by launches, and the kernel is not tried again."""
    for n, _, graph, _, same, _ in child([[n, 1] for n in
                                          (1000, 3000, 8193, 100003, -1)]):
        assert graph == [1, 0], n
        assert same, n


def _time_runs(vc, n, k, T=50):
    import torch
    rng = np.random.default_rng(3)
    obs = dev(np.cumsum(rng.normal(0, 0.1, (T, 2)), 0))
    pfs = [vc.ParticleFilter(n, 32, vc.SYSTEMATIC, 0.5, seed=1 + i,
                             max_steps=T) for i in range(k)]
    best = np.inf
    for _ in range(9):
        torch.cuda.synchronize()
        t = time.perf_counter()
        for pf in pfs:
            vc.call("vsmc_cuda_pf_run_device", pf.handle, T, obs.data_ptr())
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    for pf in pfs:
        pf.close()
    return best


@pytest.mark.parametrize("n", [20000, 100003, 155000, 200000, 300000])
def test_two_filters_overlap(vc, n):
    """Two filters on streams of their own take less than 1.6 times one (1.05
    to 1.25 where the chip has room for both; 2 where one holds it all)."""
    one, two = _time_runs(vc, n, 1), _time_runs(vc, n, 2)
    assert two < 1.6 * one, (one, two)


@pytest.mark.parametrize("n", [500, 5000, 50000, 400000])
def test_a_run_under_capture_is_refused(vc, n):
    """A run of several steps replays graphs of its own, so it cannot be
    captured; whichever path the size takes, it is refused, and the filter runs
    as before once the capture has ended."""
    import torch
    T = 4
    obs = np.random.default_rng(1).normal(0, 0.5, (T, 2))
    d = dev(obs)
    rt = ctypes.CDLL("libcudart.so.13")
    stream = torch.cuda.Stream()
    s = ctypes.c_void_p(stream.cuda_stream)
    pf = vc.ParticleFilter(n, 32, vc.SYSTEMATIC, 0.5, seed=1, max_steps=T,
                           stream=stream.cuda_stream)
    torch.cuda.synchronize()
    assert rt.cudaStreamBeginCapture(s, 1) == 0
    status = vc.lib().vsmc_cuda_pf_run_device(
        pf.handle, ctypes.c_size_t(T), ctypes.c_void_p(d.data_ptr()))
    graph = ctypes.c_void_p()
    rt.cudaStreamEndCapture(s, ctypes.byref(graph))
    if graph.value:
        rt.cudaGraphDestroy(graph)
    rt.cudaGetLastError()
    assert status == vc.ERR_CUDA
    got = pf.run(obs)
    pf.close()
    pf = vc.ParticleFilter(n, 32, vc.SYSTEMATIC, 0.5, seed=1, max_steps=T)
    want = pf.run(obs)
    pf.close()
    for k in want:
        assert np.array_equal(got[k], want[k]), k

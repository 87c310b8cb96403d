"""A captured call outlives later direct calls of its context: scratch that its
graph writes is neither freed nor handed back when a call with other paths,
another disparity range of the same class, another recurrence or a larger
volume of its own comes after it.  What the allocator was asked to release is
checked before the graph is replayed (and kept, filled with ones)."""
import ctypes

import numpy as np
import pytest
import torch

from thundervision_b200 import api

pytestmark = pytest.mark.gpu

W, H = 200, 72


def _context():
    live, released = {}, []

    def alloc(n, user):
        t = torch.empty(n, dtype=torch.uint8, device="cuda")
        live[t.data_ptr()] = t
        return t.data_ptr()

    def release(p, user):
        released.append(p)
        live[p].fill_(255)  # kept: its memory is not used by anyone else

    c = api.Context(0)
    c.set_allocator(alloc, release)
    return c, live, released


def _pair(w=W, h=H, seed=11):
    rng = np.random.default_rng(seed)
    return [torch.from_numpy(rng.integers(0, 256, size=(h, w)).astype(np.uint8)).cuda() for _ in range(2)]


def _maps(out):
    return [o["disp"].to(torch.int32) for o in (out if isinstance(out, list) else [out])]


def _replay_after(warm, call, later, none_released=True):
    c, live, released = _context()
    plain = api.Context(0)
    g = torch.cuda.CUDAGraph()
    try:
        warm(c)
        call(c)
        torch.cuda.synchronize()
        with torch.cuda.graph(g):
            out = call(c)
        before = len(released)
        for f in later:
            f(c)
            torch.cuda.synchronize()
        assert released[before:] == [] or not none_released
        for o in out if isinstance(out, list) else [out]:
            o["disp"].view(torch.int16).zero_()
        g.replay()
        want = call(plain)
        torch.cuda.synchronize()
        for a, b in zip(_maps(out), _maps(want)):
            assert torch.equal(a, b)
    finally:
        del g
        torch.cuda.synchronize()
        c.close()
        plain.close()


FUSED = [dict(D=16, paths=4), dict(D=16, paths=8), dict(D=64, paths=8),
         dict(D=64, paths=8, semantics="ref_cpu", table="ref")]


def _fused(pair, D, **kw):
    return lambda c: c.stereo_sgm(*pair, D, 10, 120, lr=1, **kw)


def _frames(pair, D, **kw):
    l, r = pair
    return lambda c: c.stereo_sgm_frames([l, r, l], [r, l, r], D, 10, 120, lr=1, **kw)


@pytest.mark.parametrize("make", [_fused, _frames])
@pytest.mark.parametrize("first", [0, 1])
def test_other_calls_of_the_size(make, first):
    pair = _pair()
    _replay_after(lambda c: None, make(pair, **FUSED[first]), [make(pair, **kw) for kw in FUSED[first + 1:]])


def test_larger_call_whose_volumes_are_there():
    """The accumulating volumes hold the larger size already (penalties beyond
    the byte volumes); the byte volumes grow after the capture."""
    small, large = _pair(), _pair(2 * W, H, 3)
    _replay_after(lambda c: c.stereo_sgm(*large, 48, 10, 300), _fused(small, 48), [_fused(large, 48)])


def test_own_volume_then_a_larger_range():
    """The capture into its own volume holds no scratch that grows."""
    f = [p.float() / 255 for p in _pair()]
    plain = api.Context(0)
    small, large = plain.cost(*f, 32), plain.cost(*f, 56)
    s_small, s_large = torch.empty_like(small), torch.empty_like(large)
    _replay_after(lambda c: None, lambda c: c.sgm(small, 0.1, 0.5, aggreg=s_small),
                  [lambda c: c.sgm(large, 0.1, 0.5, aggreg=s_large)], none_released=False)
    plain.close()


def _cudart():
    with open("/proc/self/maps") as f:
        paths = {ln.split()[-1] for ln in f if "libcudart.so" in ln}
    return ctypes.CDLL(sorted(paths)[0])


def test_capture_behind_a_queued_call():
    """A capture begun while the warm-up call is still queued, as a C caller may
    (torch's own capture waits first): the graph gets the side-by-side volumes
    all the same, so the next direct call allocates its own."""
    f = [p.float() / 255 for p in _pair()]
    c, live, _ = _context()
    plain = api.Context(0)
    rt = _cudart()
    graph, gexec = ctypes.c_void_p(), ctypes.c_void_p()
    try:
        cost = plain.cost(*f, 32)
        own = torch.empty_like(cost)
        want = plain.sgm(cost, 0.1, 0.5)["disp"].to(torch.int32)
        c.sgm(cost, 0.1, 0.5)
        s = torch.cuda.Stream()
        st = ctypes.c_void_p(s.cuda_stream)
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            c.sgm(cost, 0.1, 0.5)  # leaves a cached output block to the captured call
            torch.cuda._sleep(400_000_000)
            c.sgm(cost, 0.1, 0.5)
            assert not s.query()
            assert rt.cudaStreamBeginCapture(st, 0) == 0
            out = c.sgm(cost, 0.1, 0.5)["disp"]
            assert rt.cudaStreamEndCapture(st, ctypes.byref(graph)) == 0
            assert rt.cudaGraphInstantiate(ctypes.byref(gexec), graph, ctypes.c_ulonglong(0)) == 0
            n = len(live)
            direct = c.sgm(cost, 0.1, 0.5, aggreg=own)["disp"]
            assert len(live) == n + 1
            assert rt.cudaGraphLaunch(gexec, st) == 0
        torch.cuda.synchronize()
        assert torch.equal(out.to(torch.int32), want)
        assert torch.equal(direct.to(torch.int32), want)
    finally:
        torch.cuda.synchronize()
        if gexec:
            rt.cudaGraphExecDestroy(gexec)
        if graph:
            rt.cudaGraphDestroy(graph)
        c.close()
        plain.close()

"""The edge tree of a surface is built by the first signed distance asked of it, not with the surface: the memory it takes
appears then, once; first calls from several threads at once and a first call under stream capture give the results of
any later call."""
import threading

import numpy as np
import pytest
import torch

from warpsphboundaries_b200 import _lib, workloads
from warpsphboundaries_b200.scene import SurfaceRep

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def _surface(n, support, seed=4):
    rep = SurfaceRep.polygon(workloads.star(np.random.default_rng(seed), (0.1, 0.2), 0.8, n, jitter=0.0), conditioned=False)
    return rep.native(support, DEV)


def _distance(ns, P, out, stream):
    d, cp, nl, ed = out
    _lib.check(_lib.lib.wsb_signed_distance(ns.handle, _lib.ptr(P), len(P), 0.1, _lib.ptr(d), _lib.ptr(cp), _lib.ptr(nl),
                                            _lib.ptr(ed), _lib.c_void_p(stream.cuda_stream)), "wsb_signed_distance")


def _outputs(m):
    return [torch.empty(s, dtype=t, device=DEV) for s, t in (((m,), torch.float64), ((m, 2), torch.float64),
                                                             ((m, 2), torch.float64), ((m,), torch.int32))]


def _points(m):
    g = torch.Generator(device=DEV)
    g.manual_seed(5)
    return 3 * torch.rand((m, 2), dtype=torch.float64, device=DEV, generator=g) - 1.5


def test_no_tree_before_the_first_distance():
    n = 400_000                                                   # 36 bytes an edge and the boxes: 16 MB
    ns, P = _surface(n, 0.01), _points(64)
    outs = [_outputs(64) for _ in range(2)]
    free = []
    for out in (None, outs[0], outs[1]):
        if out is not None:
            _distance(ns, P, out, torch.cuda.current_stream())
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[1] >= 36 * n and free[1] == free[2]
    assert all(torch.equal(a, b) for a, b in zip(*outs))


def test_first_calls_of_several_threads():
    P, errors = _points(5000), []
    ns = _surface(3000, 0.05)
    outs = [_outputs(len(P)) for _ in range(8)]
    torch.cuda.synchronize()
    gate = threading.Barrier(len(outs))

    def work(out):
        try:
            st = torch.cuda.Stream()
            gate.wait(timeout=30)
            _distance(ns, P, out, st)
            st.synchronize()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(o,)) for o in outs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    again = _outputs(len(P))
    _distance(ns, P, again, torch.cuda.current_stream())
    for out in outs:
        assert all(torch.equal(a, b) for a, b in zip(out, again))


def test_first_call_under_capture():
    P = _points(1000)
    ns, out, again = _surface(700, 0.05), _outputs(1000), _outputs(1000)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _distance(ns, P, out, torch.cuda.current_stream())
    graph.replay()
    _distance(ns, P, again, torch.cuda.current_stream())
    assert all(torch.equal(a, b) for a, b in zip(out, again))

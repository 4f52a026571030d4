"""Kept constants (scalar parameters, the shared record's indices): several streams and threads, more values than are
kept, growing element counts, and calls captured in a graph."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(E, k6, alpha, explicit):
    import torch
    from pyfe3d_gb300 import batch
    from pyfe3d_gb300.shellprop import isotropic_plate_records
    rng = np.random.default_rng(E)
    x = np.zeros((E, 3, 3))
    x[:, :, :2] = np.array([[0, 0], [1, 0], [0, 1]]) + rng.uniform(-0.2, 0.2, (E, 3, 2))
    cdof = 6 * np.arange(3 * E, dtype=np.int64).reshape(E, 3)
    v = torch.zeros(324 * E, dtype=torch.float64, device='cuda')
    kw = dict(k6rot=k6, alpha=alpha)
    if explicit:
        kw = dict(k6rot=np.full(E, k6), alpha=np.full(E, alpha), pid=np.zeros(E, np.int32))
    batch.tria3r_update_KC0(None, None, v, x.ravel(), cdof, 324 * np.arange(E, dtype=np.int64),
                            isotropic_plate_records(0.01, 70e9, 0.3), update_KC0v_only=1, **kw)
    return v


def test_kept_constants_match_given_arrays(gpulib):
    import torch
    bad = []

    def work(seed):
        rng = np.random.default_rng(seed)
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(40):
                E, k6, alpha = int(rng.integers(2, 3000)), float(rng.uniform(1, 200)), float(rng.uniform(0.1, 1))
                if not torch.equal(_run(E, k6, alpha, False), _run(E, k6, alpha, True)):
                    bad.append((seed, i))
    threads = [threading.Thread(target=work, args=(s,)) for s in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    from pyfe3d_gb300 import _lib
    assert len(_lib._constants._kept) <= 64


def test_captured_call_keeps_its_own_constants(gpulib):
    import torch
    from pyfe3d_gb300 import batch
    from pyfe3d_gb300.shellprop import isotropic_plate_records
    E = 50
    want = _run(E, 77., 0.5, True)
    rng = np.random.default_rng(E)
    x = np.zeros((E, 3, 3))
    x[:, :, :2] = np.array([[0, 0], [1, 0], [0, 1]]) + rng.uniform(-0.2, 0.2, (E, 3, 2))
    d = [torch.from_numpy(a).cuda() for a in (x.ravel(), 6 * np.arange(3 * E, dtype=np.int64).reshape(E, 3),
                                              324 * np.arange(E, dtype=np.int64),
                                              isotropic_plate_records(0.01, 70e9, 0.3))]
    v = torch.zeros_like(want)
    call = lambda: batch.tria3r_update_KC0(None, None, v, d[0], d[1], d[2], d[3], k6rot=77., alpha=0.5,  # noqa: E731
                                           update_KC0v_only=1, check=False)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        call()
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        v.zero_()
        call()
    for i in range(70):  # more values than are kept
        _run(3, 100. + i, 0.3, False)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(v, want)

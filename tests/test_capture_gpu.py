"""Exact searches and graph capture: a captured call does not grow its workspace, and the operand copy that a later call of one
thread lays out does not disturb another thread's capture."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(n, dim, nq, k):
    import torch
    from annvedi_b200.linear import LinearIndex
    rng = np.random.default_rng(n)
    ix = LinearIndex(device=0, mode="exact")
    ix.fit(torch.from_numpy(rng.standard_normal((n, dim)).astype(np.float32)).cuda())
    q = torch.from_numpy(rng.standard_normal((nq, dim)).astype(np.float32)).cuda()
    return ix, q, torch.empty(nq, k, dtype=torch.int64, device="cuda"), torch.empty(nq, k, device="cuda")


def test_captured_call_keeps_to_its_workspace(cuda):
    """A workspace sized by calls of the scan; then the index begins to prune (by calls with another workspace); then the
    capture with the first one."""
    import torch
    from annvedi_b200.linear import Workspace
    ix, q, ids, d = _setup(40000, 64, 6, 10)
    ws, other = Workspace(0), Workspace(0)
    s = torch.cuda.Stream()

    def call(w):
        ix.search(q, 10, workspace=w, out_ids=ids, out_dists=d, stream=s)

    with torch.cuda.stream(s):
        call(ws)
    ix.search_tc(q[:1], 1)
    with torch.cuda.stream(s):
        for _ in range(3):
            call(other)
    torch.cuda.synchronize()
    assert ix.get_prune_stats()["passes"] >= 1
    want = ids.clone(), d.clone()
    size = ws.nbytes()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        call(ws)
    assert ws.nbytes() == size
    ids.zero_(), d.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(ids, want[0]) and torch.equal(d, want[1])


def test_layout_beside_another_threads_capture(cuda):
    import torch
    from annvedi_b200.linear import Workspace
    ix, q, ids, d = _setup(60000, 64, 6, 10)
    ws = Workspace(0)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        ix.search(q, 10, workspace=ws, out_ids=ids, out_dists=d, stream=s)  # the scan, its scratch sized
    torch.cuda.synchronize()
    want = ids.clone(), d.clone()
    x = torch.ones(1000, device="cuda")
    errors = []

    def search():
        try:
            for _ in range(30):  # (the layout comes with the savings of about a dozen calls)
                ix.search(q, 10, workspace=ws, out_ids=ids, out_dists=d, stream=s)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = x * 2
        t = threading.Thread(target=search)
        t.start()
        t.join()
        z = y + 1
    assert not errors, errors
    g.replay()
    torch.cuda.synchronize()
    assert (z == 3).all()
    assert ix.get_prune_stats()["passes"] >= 1
    assert torch.equal(ids, want[0]) and torch.equal(d, want[1])

"""Plans and workspaces that calls keep for the next one: graph captures, streams and threads must not see each
other's."""
import threading

import pytest
import torch

import ae296_b200 as L

pytestmark = pytest.mark.gpu

N, H = 9, 512


def _op_inputs(T, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(T, H, generator=g).half().cuda()
    wa = (torch.randn(N, 1, 16, H, generator=g) / H ** 0.5).half().cuda()
    wb = (torch.randn(N, 1, H, 16, generator=g) / 4).half().cuda()
    return x, wa, wb, [torch.randint(0, N, (T,), generator=g).cuda() for _ in range(2)]


def _once(x, wa, wb, ids):
    """The same op with a plan of its own: the bits every kept-plan call must give."""
    y = torch.zeros(x.shape[0], H, dtype=x.dtype, device="cuda")
    ws = torch.empty(L.add_lora_bgmv_workspace_bytes(x.shape[0], N, H), dtype=torch.uint8, device="cuda")
    L.add_lora_bgmv_once(y, x, wa, wb, ids, 0, 1.0, ws)
    return y


def _op(y, x, wa, wb, ids):
    y.zero_()
    L.add_lora_bgmv(y, x, wa, wb, ids, 0, 1.0)


def _capture(s, fn):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        fn()
    return g


def test_operator_eager_replay_eager_on_one_stream():
    """A replay rebuilds its own plan and not the one that eager calls of the stream keep."""
    x, wa, wb, (ids1, ids2) = _op_inputs(40, 1)
    want1, want2 = _once(x, wa, wb, ids1), _once(x, wa, wb, ids2)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    ye, yg = torch.zeros_like(want1), torch.zeros_like(want1)
    with torch.cuda.stream(s):
        _op(ye, x, wa, wb, ids1)
        g = _capture(s, lambda: _op(yg, x, wa, wb, ids2))
        _op(ye, x, wa, wb, ids1)
        g.replay()
        _op(ye, x, wa, wb, ids1)
    torch.cuda.synchronize()
    assert torch.equal(yg, want2) and torch.equal(ye, want1)
    ids2.copy_(ids1)                                       # a replay follows the contents of its index tensor
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(yg, want1)


def test_operator_graphs_of_growing_batches_keep_their_memory():
    """Larger calls on the stream, eager and captured, leave an earlier graph its plan and workspace."""
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graphs = []
    with torch.cuda.stream(s):
        for T in (8, 60, 300):
            x, wa, wb, (ids, _) = _op_inputs(T, T)
            y, want = torch.zeros(T, H, dtype=x.dtype, device="cuda"), _once(x, wa, wb, ids)
            _op(y, x, wa, wb, ids)                         # the usual warm-up
            graphs.append((_capture(s, lambda: _op(y, x, wa, wb, ids)), y, want, (x, wa, wb, ids)))
        # whatever was given back is in use by others now
        others = [torch.full((n,), 7, dtype=torch.int32, device="cuda") for n in (1 << 10, 1 << 14, 1 << 18, 1 << 20) for _ in range(8)]
        for _ in range(2):
            for g, y, _, _ in graphs:
                y.zero_()
                g.replay()
    torch.cuda.synchronize()
    for _, y, want, _ in graphs:
        assert torch.equal(y, want)
    assert all(bool((o == 7).all()) for o in others)


def test_operator_called_by_threads_on_one_stream():
    """Threads that share a stream share its plan: no call may run with the ids of another thread's, also while
    the batches grow."""
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    jobs = []
    for k in range(4):
        x, wa, wb, (ids, _) = _op_inputs(24 + 8 * k, 50 + k)
        jobs.append((x, wa, wb, ids, _once(x, wa, wb, ids)))
    torch.cuda.synchronize()
    wrong, errors = [], []

    def work(x, wa, wb, ids, want):
        try:
            with torch.cuda.stream(s):
                ys = [torch.zeros_like(want) for _ in range(400)]
                for y in ys:
                    L.add_lora_bgmv(y, x, wa, wb, ids, 0, 1.0)
                s.synchronize()
                wrong.append(sum(not torch.equal(y, want) for y in ys))
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and wrong == [0] * len(jobs)

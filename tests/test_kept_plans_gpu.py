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


# ---- the layer object ----------------------------------------------------------------------------
def _layer_object(T=24):
    torch.manual_seed(3)
    obj = L.Lora_GPU({"n_layers": 2, "batch_size": 32, "lora_rank": 16, "hidden_dim": H, "tp_degree": 1,
                      "max_prefill_batch_size": 6})
    x = torch.randn(T, H, device="cuda").half()
    ids = [torch.randint(0, 32, (T,), device="cuda", generator=torch.Generator("cuda").manual_seed(k)) for k in range(2)]

    def want(i):
        y = torch.zeros_like(x)
        ws = torch.empty(L.add_lora_bgmv_workspace_bytes(T, 32, H), dtype=torch.uint8, device="cuda")
        L.add_lora_bgmv_once(y, x, obj.q_down, obj.q_up, ids[i], 1, 1.0, ws)
        return y.float()

    def same(got, i):                     # the fused call cuts the split-K sums elsewhere: one ulp
        w = want(i)
        torch.cuda.synchronize()
        return bool(((got.float() - w).abs() <= 2.0 ** -10 * w.abs() + 2.0 ** -24).all())

    return obj, x, ids, same


def test_layer_object_eager_steps_after_replays():
    """A graph captured with one set of indices, eager steps with another before and after its replay."""
    obj, x, (a, b), same = _layer_object()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    out = {}
    with torch.cuda.stream(s):
        obj.set_indices(a)
        obj.invoke_one_layer_q(x, 1)                       # warm-up
        obj.set_indices(a)
        g = _capture(s, lambda: out.update(g=obj.invoke_one_layer_q(x, 1)))
        obj.set_indices(b)
        before = obj.invoke_one_layer_q(x, 1)
        g.replay()
        after = obj.invoke_one_layer_q(x, 1)
    torch.cuda.synchronize()
    assert same(before, 1) and same(out["g"], 0) and same(after, 1)


def test_layer_object_eager_step_before_the_first_replay():
    """A plan that was only captured has not been built: the eager step makes its own."""
    obj, x, (a, b), same = _layer_object()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        obj.set_indices(a)
        obj.invoke_one_layer_q(x, 1)
        obj.set_indices(b)
        _capture(s, lambda: obj.invoke_one_layer_q(x, 1))
        eager = obj.invoke_one_layer_q(x, 1)
    torch.cuda.synchronize()
    assert same(eager, 1)


def test_layer_object_graph_keeps_its_indices():
    """set_indices and an eager step leave a captured graph with the indices of its capture."""
    obj, x, (a, b), same = _layer_object()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    out = {}
    with torch.cuda.stream(s):
        obj.set_indices(a)
        obj.invoke_one_layer_q(x, 1)                       # the plan exists: the capture must build it again
        g = _capture(s, lambda: out.update(g=obj.invoke_one_layer_q(x, 1)))
        obj.set_indices(b)
        obj.invoke_one_layer_q(x, 1)
        g.replay()
    torch.cuda.synchronize()
    assert same(out["g"], 0)


def test_layer_object_on_two_streams():
    """Steps with different indices in flight on two streams have plans and workspaces of their own."""
    obj, x, (a, b), same = _layer_object()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    got = [[], []]
    for _ in range(20):
        for i, ids in enumerate((a, b)):
            with torch.cuda.stream(streams[i]):
                obj.set_indices(ids)
                got[i] += [obj.invoke_one_layer_q(x, 1) for _ in range(3)]
    torch.cuda.synchronize()
    batches = {id(k.batch) for k in obj._kept.values()}
    assert len(batches) == 2
    assert all(same(y, i) for i in range(2) for y in got[i])


def test_layer_object_prefill_shape_only_captured():
    """As above for prefill: a shape whose segment table was only captured is built by the eager call."""
    obj, _, _, _ = _layer_object()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    xs = [torch.randn(*shape, H, device="cuda").half() for shape in ((2, 60), (3, 40))]
    with torch.cuda.stream(s):
        obj.invoke_one_layer_q(xs[0], 1, prefill=True)
        _capture(s, lambda: obj.invoke_one_layer_q(xs[1], 1, prefill=True))
        got = obj.invoke_one_layer_q(xs[1], 1, prefill=True)
    torch.cuda.synchronize()
    for i in range(3):
        v = (xs[1][i].float() @ obj.q_down_prefill[i, 1].float().t()).half().float()
        want = v @ obj.q_up_prefill[i, 1].float().t()
        rms = float(want.pow(2).mean().sqrt())
        # one rounding of the result, and of an intermediate that may fall on the other side of a tie
        assert float((got[i].float() - want).abs().max()) <= 2e-3 * rms + float(want.abs().max()) * 2 ** -10


def test_layer_object_parts_of_a_captured_or_foreign_q_call_are_not_handed_out():
    """k after a q call that was only captured, or that ran on another stream: its own computation."""
    obj, x, (a, _), _ = _layer_object()
    obj.set_indices(a)
    want = obj.invoke_one_layer_k(x, 1).clone()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        obj.invoke_one_layer_q(x, 0)                       # warm-up
        part = {}

        def q():
            obj.invoke_one_layer_q(x, 1)
            part["k"] = obj._fused[1][1]

        g = _capture(s, q)
        k = obj.invoke_one_layer_k(x, 1)
    torch.cuda.synchronize()
    assert k.data_ptr() != part["k"].data_ptr() and torch.equal(k, want)
    obj.invoke_one_layer_q(x, 1)
    other = obj._fused[1][1]
    with torch.cuda.stream(s):
        k = obj.invoke_one_layer_k(x, 1)
    torch.cuda.synchronize()
    assert k.data_ptr() != other.data_ptr() and torch.equal(k, want)


def test_layer_object_parts_of_a_q_call_with_other_indices_are_not_handed_out():
    obj, x, (a, b), _ = _layer_object()
    obj.set_indices(b)
    want = obj.invoke_one_layer_k(x, 1).clone()
    obj.set_indices(a)
    obj.invoke_one_layer_q(x, 1)
    obj.set_indices(b)
    assert torch.equal(obj.invoke_one_layer_k(x, 1), want)

"""GPU parity of the decode BGMV path against the CPU oracle, through the C ABI."""
import numpy as np
import pytest
import torch

import ae296_b200 as L
from ae296_b200 import _lib
from lora_testlib import TOL, Case, rel_err
from oracle import lora_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 2, 31, 33])
@pytest.mark.parametrize("r", [8, 16, 64])
@pytest.mark.parametrize("H", [128, 4096])
def test_tiny_exhaustive(T, r, H):
    c = Case(T, 5, H, H, r, "fp16", dense=False, seed=T * 100 + r + H)
    want = c.oracle_delta(1)
    y32 = c.run(1, y_dtype=torch.float32)
    assert rel_err(y32.double().cpu().numpy(), want) <= TOL
    y16 = c.run(1)
    # the low-precision output is the single rounding of the fp32 result
    assert torch.equal(y16, y32.to(torch.float16))
    # a second run is bit-identical (fixed-order split-K reduction, no float atomics)
    assert torch.equal(c.run(1, y_dtype=torch.float32), y32)


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("dense", [False, True])
def test_mixed_ranks_both_layouts(dtype, dense):
    c = Case(96, 24, 1024, 768, [8, 16, 32, 64], dtype, dense=dense, seed=7, zipf=1.0)
    for layer in (0, 1):
        want = c.oracle_delta(layer)
        y32 = c.run(layer, y_dtype=torch.float32)
        assert rel_err(y32.double().cpu().numpy(), want) <= TOL
        assert torch.equal(c.run(layer), y32.to(c.tdt))


def test_dense_pool_ranks_not_multiple_of_8_and_garbage_padding():
    c = Case(40, 6, 512, 512, np.array([3, 12, 20, 33, 50, 64], np.int32), "fp16", dense=True, seed=3)
    # poison the unused rows/columns of the dense pool: they must never be read into the result
    for a in range(c.N):
        r = int(c.ranks[a])
        c.pool.wa[a, :, r:, :] = float("nan")
        c.pool.wb[a, :, :, r:] = float("nan")
    y32 = c.run(0, y_dtype=torch.float32)
    assert rel_err(y32.double().cpu().numpy(), c.oracle_delta(0)) <= TOL


@pytest.mark.parametrize("h_in,h_out", [(128, 128), (640, 1152), (1152, 640), (256, 3072), (2048, 8192), (8192, 1024)])
@pytest.mark.parametrize("T,N,ranks,dtype", [(1, 1, [64], "bf16"), (8, 1, [8], "fp16"), (5, 2, [32, 16], "bf16"), (10, 4, [8, 64, 16, 32], "fp16")])
def test_few_tokens_in_one_launch(T, N, ranks, dtype, h_in, h_out):
    """The cluster kernel: every rank, one to eight tokens a segment, slices of h_in and h_out that are empty or
    uneven over the eight CTAs, two projections; and the streaming kernels on the same rows (a batch too large
    for the cluster route) to the precision both keep v in."""
    ids = np.arange(T) % N
    c = Case(T, N, h_in, h_out, np.array(ranks, np.int32), dtype, seed=T + h_in, ids=ids)
    y32 = c.run(1, y_dtype=torch.float32)
    assert rel_err(y32.double().cpu().numpy(), c.oracle_delta(1)) <= TOL
    assert torch.equal(c.run(1), y32.to(c.tdt))
    assert torch.equal(c.run(1, y_dtype=torch.float32), y32)
    if dtype == "fp16":                   # (a bf16 tie that falls the other way is larger than the bound)
        assert rel_err(c.run(1, y_dtype=torch.float32, flags=L.MID_ROUND).double().cpu().numpy(), c.oracle_delta(1, mid_round=dtype)) <= TOL
    ys = [torch.ones(T, h_out, dtype=c.tdt, device="cuda") for _ in range(2)]
    L.LoraBatch(T, N, h_in, 2).set_ids(c.ids_dev, c.pool).apply([(c.x, y, c.pool) for y in ys], 1)
    # (twenty items may be past the cluster route: one rounding of y + delta, and the bound derived below)
    ulp = 2.0 ** (-8 if dtype == "bf16" else -11)
    assert torch.equal(ys[0], ys[1])
    assert bool(((ys[0].float() - (y32 + 1)).abs() <= ulp * (y32 + 1).abs() + 1e-4 * y32.pow(2).mean().sqrt()).all())
    reps = 200 // T + 1
    big = torch.zeros(reps * T, h_out, dtype=torch.float32, device="cuda")
    L.LoraBatch(reps * T, N, h_in, 1).set_ids(c.ids_dev.repeat(reps), c.pool).apply([(c.x.repeat(reps, 1), big, c.pool)], 1)
    # The two differ in the order of their fp32 sums, and in what the 16-bit halves of v then drop: at most 2^-17 |v| each
    # in bf16, so 2^-16 sum |v||b| between them if all fell one way (sum |v||b| is at most about 8 times the RMS of
    # y = sum v b for r <= 64: 1.2e-4), and an eighth of that for errors of either sign.
    assert rel_err(big[:T].double().cpu().numpy(), y32.double().cpu().numpy()) <= 1e-4


def test_few_tokens_with_y_in_the_memory_of_x():
    """y += delta(x) with y the same rows as x: every projection still sees the old x."""
    c = Case(6, 3, 512, 512, [16], "fp16", seed=77)
    want = O.round_to(c.x_cpu.double().numpy() + c.oracle_delta(0), "fp16")
    y2 = torch.zeros(6, 512, dtype=torch.float16, device="cuda")
    c_x = c.x.clone()
    L.LoraBatch(6, 3, 512, 2).set_ids(c.ids_dev, c.pool).apply([(c_x, c_x, c.pool), (c_x, y2, c.pool)], 0)
    assert np.abs(c_x.double().cpu().numpy() - want).max() <= np.abs(want).max() * 2 ** -10
    delta = c.oracle_delta(0)
    assert np.abs(y2.double().cpu().numpy() - delta).max() <= np.abs(delta).max() * 2 ** -10


@pytest.mark.parametrize("r_max,ranks", [(8, [1, 7, 8]), (16, [9, 15, 16, 2]), (24, [24, 17, 8, 3]), (40, [40, 33, 16, 5]),
                                         (64, [63, 31, 12, 64])])
@pytest.mark.parametrize("T,h_in,h_out,dtype", [(1, 128, 640, "fp16"), (9, 640, 128, "bf16"), (70, 2176, 2432, "fp16")])
def test_padded_dense_pools_of_any_rank(r_max, ranks, T, h_in, h_out, dtype):
    """Dense pools R that hold ranks below R: every rank class and its edges, R itself below its class, partial
    units and partial super-chunks, one to full work segments; what lies beyond an adapter's rank is NaN."""
    c = Case(T, len(ranks), h_in, h_out, np.array(ranks, np.int32), dtype, dense=True, seed=r_max + T)
    assert c.pool.r_pool == r_max
    for a, r in enumerate(ranks):
        c.pool.wa[a, :, r:, :] = float("nan")
        c.pool.wb[a, :, :, r:] = float("nan")
    for layer in (0, c.n_layers - 1):
        y32 = c.run(layer, y_dtype=torch.float32)
        assert rel_err(y32.double().cpu().numpy(), c.oracle_delta(layer)) <= TOL
        assert torch.equal(c.run(layer), y32.to(c.tdt))


def test_accumulates_into_y_with_strides_and_canaries():
    c = Case(37, 9, 640, 384, [16, 32], "bf16", seed=11)
    g = torch.Generator().manual_seed(5)
    pad = 16
    ybig = torch.randn(c.T + 2, c.h_out + 2 * pad, generator=g).to(torch.bfloat16).cuda()
    before = ybig.clone()
    xbig = torch.full((c.T, c.h_in + 24), 7.0, dtype=torch.bfloat16, device="cuda")
    xbig[:, :c.h_in] = c.x
    yv = ybig[1:-1, pad:pad + c.h_out]
    batch = L.LoraBatch(c.T, c.N, c.h_in, 1).set_ids(c.ids_dev, c.pool)
    batch.apply([(xbig[:, :c.h_in], yv, c.pool)], 1)
    torch.cuda.synchronize()
    want = O.round_to(before[1:-1, pad:pad + c.h_out].double().cpu().numpy() + c.oracle_delta(1), "bf16")
    got = yv.double().cpu().numpy()
    rms = np.sqrt((want ** 2).mean())
    # one bf16 rounding of (y + delta): within half an ulp of the exact sum plus the fp32 error
    assert np.abs(got - want).max() <= np.abs(want).max() * 2 ** -8 + TOL * rms
    mask = torch.ones_like(ybig, dtype=torch.bool)
    mask[1:-1, pad:pad + c.h_out] = False
    assert torch.equal(ybig[mask], before[mask]), "bytes outside the y view were written"


def test_reference_call_signature_int64_ids():
    c = Case(32, 8, 4096, 4096, 16, "fp16", dense=True, seed=2960)
    y = torch.zeros(c.T, c.h_out, dtype=torch.float16, device="cuda")
    ret = L.add_lora_bgmv(y, c.x, c.pool.wa, c.pool.wb, c.ids_dev.long(), 1, 2.0)
    torch.cuda.synchronize()
    assert ret is None
    want = O.lora_delta(c.x_cpu.double().numpy(), lambda a: c.A[a][1].double().numpy(),
                        lambda a: c.B[a][1].double().numpy(), c.ids, np.full(c.N, 2.0))
    got = y.double().cpu().numpy()
    rms = np.sqrt((want ** 2).mean())
    assert np.abs(got - want).max() <= TOL * rms + np.abs(want).max() * 2 ** -11


def test_mid_round_flag_matches_bmm_rounding():
    c = Case(64, 4, 512, 512, 32, "fp16", seed=9, ids=np.repeat(np.arange(4), 16))
    y32 = c.run(0, y_dtype=torch.float32, flags=L.MID_ROUND)
    assert rel_err(y32.double().cpu().numpy(), c.oracle_delta(0, mid_round="fp16")) <= TOL


def test_fused_qkv_equals_separate_calls():
    c = Case(48, 12, 1024, 1024, [8, 64], "fp16", seed=21, zipf=1.0)
    k = Case(48, 12, 1024, 256, c.ranks, "fp16", seed=22, ids=c.ids)
    ys = [torch.zeros(48, h, dtype=torch.float16, device="cuda") for h in (1024, 256, 1024)]
    batch = L.LoraBatch(48, 12, 1024, 3).set_ids(c.ids_dev, c.pool)
    batch.apply([(c.x, ys[0], c.pool), (c.x, ys[1], k.pool), (c.x, ys[2], c.pool)], 1)
    torch.cuda.synchronize()
    batch.workspace.check()

    def close(a, b):
        # the fused call cuts the split-K sums at other places than a single-projection call,
        # so the fp32 sums may differ in their last bits: allow one fp16 ulp of the result
        a, b = a.float(), b.float()
        return bool(((a - b).abs() <= 2.0 ** -10 * b.abs().clamp_min(2.0 ** -6)).all())

    assert close(ys[0], c.run(1))
    assert close(ys[2], ys[0])
    k.x, k.x_cpu = c.x, c.x_cpu
    assert close(ys[1], k.run(1))


def test_outputs_side_by_side_in_one_buffer():
    """q | k | v as column ranges of one [T, sum(h_out)] block (row pitch larger than the width), x as
    one of two activations that share a buffer: same bits as separate contiguous tensors, nothing
    written outside the ranges.  Decode kernels and, with tall runs, the tile kernel."""
    for tiles, ids in ((False, None), (True, np.concatenate([np.arange(40) % 6, np.repeat([7, 2], [128, 70])]).astype(np.int32))):
        T = 48 if ids is None else len(ids)
        c = Case(T, 12, 1024, 1024, [16, 64], "bf16", seed=31, zipf=1.0 if ids is None else None, ids=ids)
        k = Case(T, 12, 1024, 256, c.ranks, "bf16", seed=32, ids=c.ids)
        pools, widths = [c.pool, k.pool, c.pool], [1024, 256, 1024]
        xx = torch.zeros(2, T, 1024, dtype=torch.bfloat16, device="cuda")
        xx[1].copy_(c.x)
        g = torch.Generator().manual_seed(9)
        block = torch.randn(T, sum(widths) + 64, generator=g).to(torch.bfloat16).cuda()     # 64 canary columns
        sep = [block[:, o:o + w].clone() for o, w in zip((0, 1024, 1280), widths)]
        before = block.clone()
        views = [block[:, o:o + w] for o, w in zip((0, 1024, 1280), widths)]
        batch = L.LoraBatch(T, 12, 1024, 3).set_ids(c.ids_dev, c.pool, tiles=tiles)
        batch.apply([(xx[1], v, p) for v, p in zip(views, pools)], 1)
        batch.apply([(c.x, y, p) for y, p in zip(sep, pools)], 1)
        torch.cuda.synchronize()
        batch.workspace.check()
        for v, y in zip(views, sep):
            assert torch.equal(v, y)
        assert torch.equal(block[:, sum(widths):], before[:, sum(widths):])
        assert not torch.equal(views[0], before[:, :1024])


def test_errors_are_raised_not_swallowed():
    c = Case(8, 4, 128, 128, 8, "fp16", seed=1)
    bad = c.ids_dev.clone()
    bad[3] = 4                      # == N: out of range
    batch = L.LoraBatch(8, 4, 128, 1)
    batch.plan.build(bad, L.adapters_of(c.pool))
    with pytest.raises(L.LoraError) as e:
        batch.plan.read()
    assert e.value.code == -8
    # such a plan applies nothing
    y = torch.zeros(8, 128, dtype=torch.float16, device="cuda")
    batch.apply([(c.x, y, c.pool)], 0)
    torch.cuda.synchronize()
    assert not y.any()
    with pytest.raises(L.LoraError):
        batch.set_ids(c.ids_dev, c.pool).apply([(c.x, y, c.pool)], 5)       # layer out of range
    with pytest.raises(ValueError):
        L.add_lora_bgmv(y.cpu(), c.x.cpu(), c.pool.wa.cpu(), c.pool.wb.cpu(), c.ids_dev.cpu(), 0, 1.0)


@pytest.mark.parametrize("host_type", [np.int64, np.float32])
def test_pools_whose_host_ranks_have_another_type(host_type):
    c = Case(20, 5, 256, 384, [8, 16, 64], "fp16", seed=4, n_layers=1)
    want = c.run(0)
    c.pool.ranks_host = c.pool.ranks_host.astype(host_type)
    assert torch.equal(c.run(0), want)
    order = np.argsort(c.ids, kind="stable")
    starts = torch.from_numpy(np.searchsorted(c.ids[order], np.arange(6)).astype(np.int32)).cuda()
    used = torch.unique_consecutive(starts)
    owner = c.ids_dev[torch.from_numpy(order).cuda()][used[:-1].long()]
    y = torch.zeros_like(want)
    L.LoraBatch(20, 5, 256, 1).set_segments(used, owner, 20, c.pool).apply([(c.x[torch.from_numpy(order).cuda()], y, c.pool)], 0)
    assert torch.equal(y, want[torch.from_numpy(order).cuda()])


def test_numbers_of_other_types_as_layer_and_scale():
    c = Case(7, 4, 128, 256, 16, "fp16", dense=True, seed=6)
    for op in (L.add_lora_bgmv, L.add_lora_bgmv_static):
        ys = [torch.zeros(7, 256, dtype=torch.float16, device="cuda") for _ in range(3)]
        for y, layer, scale in zip(ys, (1, 1.0, np.float32(1)), (0.5, np.float32(0.5), "0.5")):
            op(y, c.x, c.pool.wa, c.pool.wb, c.ids_dev, layer, scale)
        assert ys[0].any() and torch.equal(ys[1], ys[0]) and torch.equal(ys[2], ys[0])


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
def test_delta_then_add_mode(dtype):
    """The reference adds the 16-bit delta to the projection in 16-bit arithmetic (q += q_lora)."""
    c = Case(70, 12, 1024, 768, [8, 16, 32, 64], dtype, seed=77, zipf=1.0)
    # y starting at zero (how the reference calls the op): identical to the default mode
    assert torch.equal(c.run(1, flags=L.DELTA_THEN_ADD), c.run(1))
    # y starting elsewhere: round(delta) added in the I/O type, the oracle's delta_then_add
    g = torch.Generator().manual_seed(3)
    y0 = torch.randn(c.T, c.h_out, generator=g).to(c.tdt).cuda()
    got = c.run(1, y0=y0, flags=L.DELTA_THEN_ADD).double().cpu().numpy()
    delta = O.round_to(c.oracle_delta(1), dtype)
    want = O.delta_then_add(y0.double().cpu().numpy(), delta, dtype)
    ulp = 2.0 ** (-10 if dtype == "fp16" else -7)
    assert np.abs(got - want).max() <= ulp * np.abs(want).max()
    assert (got != want).mean() < 0.02          # only ties of the delta's own rounding may differ


@pytest.mark.parametrize("T,N,h_in,h_out,ranks,zipf,dtype", [
    (256, 128, 4096, 4096, [8, 16, 32, 64], 1.0, "fp16"),      # decode batch of the 7B workload
    (512, 96, 8192, 1024, 64, 1.2, "bf16"),                    # GQA k/v shapes of the 70B workload
    (512, 96, 8192, 8192, 64, 1.2, "bf16"),                    # its q/o shapes: 64 units per segment
])
def test_full_size_decode_segments_spanning_many_ctas(T, N, h_in, h_out, ranks, zipf, dtype):
    """At these sizes a work segment's units are spread over several CTAs, so its intermediate is
    the sum of several split-K slots that the expand kernel's producers add up themselves."""
    c = Case(T, N, h_in, h_out, ranks, dtype, seed=11, zipf=zipf, n_layers=1)
    want = c.oracle_delta(0)
    got32 = c.run(0, y_dtype=torch.float32)
    assert rel_err(got32.double().cpu().numpy(), want) <= TOL
    # 16-bit output: the single rounding of the fp32 result; a second run is bit-identical
    got16 = c.run(0)
    assert torch.equal(got16, got32.to(c.tdt))
    assert torch.equal(c.run(0), got16)
    # linearity in x: doubling x doubles the delta; exactly so in bf16 (powers of two commute with
    # every rounding), up to the fp16 subnormals of the intermediate's lo halves in fp16
    c.x = (c.x_cpu * 2).to(c.device)
    twice = c.run(0, y_dtype=torch.float32)
    if dtype == "bf16":
        assert torch.equal(twice, got32 * 2)
    else:
        assert rel_err(twice.double().cpu().numpy(), 2 * got32.double().cpu().numpy()) <= 1e-5


def test_adapter_swapped_in_on_a_side_stream():
    """An adapter slot reloaded from pinned host memory on a side stream while the batch runs."""
    c = Case(24, 6, 512, 768, [16, 32], "fp16", seed=21)
    before = c.run(0, y_dtype=torch.float32)
    a = int(c.ids[0])
    g = torch.Generator().manual_seed(5)
    r = int(c.ranks[a])
    A_new = (torch.randn(c.n_layers, r, c.h_in, generator=g) / np.sqrt(c.h_in)).to(c.tdt).pin_memory()
    B_new = (torch.randn(c.n_layers, c.h_out, r, generator=g) / np.sqrt(r)).to(c.tdt).pin_memory()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())          # the running batch still reads the slot
    done = c.pool.load_adapter_async(a, A_new, B_new, side)
    torch.cuda.current_stream().wait_event(done)
    c.A[a], c.B[a] = A_new, B_new
    after = c.run(0, y_dtype=torch.float32)
    assert rel_err(after.double().cpu().numpy(), c.oracle_delta(0)) <= TOL
    rows = torch.from_numpy(c.ids != a).cuda()
    assert torch.equal(after[rows], before[rows])           # other adapters' tokens are untouched
    with pytest.raises(ValueError):
        c.pool.load_adapter_async(a, A_new[:, :8], B_new, side)


@pytest.mark.parametrize("kind", ["cluster", "streaming", "padded", "general", "tiles", "tiles_many"])
@pytest.mark.parametrize("y_dtype", [None, torch.float32])
def test_overwrite_equals_accumulating_into_zeros(kind, y_dtype):
    """OVERWRITE on every route: the bits that a zero-filled y gets, whatever y held; nothing outside the rows;
    zeros where the plan applies nothing."""
    T, h = {"cluster": (5, 512), "streaming": (90, 512), "padded": (90, 512), "general": (40, 328), "tiles": (300, 512),
            "tiles_many": (5000, 512)}[kind]
    ids = np.random.default_rng(T).integers(0, 6, T)
    if kind.startswith("tiles"):
        ids = np.sort(ids)
        ids[-7:] = np.arange(7) % 6                                # a few rows for the decode kernels too
    ranks = np.array([3, 12, 20, 33, 50, 64] if kind == "padded" else [8, 16, 32, 64, 16, 32], np.int32)
    c = Case(T, 6, h, h, ranks, "fp16", dense=kind == "padded", seed=T, ids=ids, n_layers=1)
    flags = _lib.OVERWRITE
    yt = c.tdt if y_dtype is None else y_dtype
    batch = L.LoraBatch(T, 6, h, 1).set_ids(c.ids_dev, c.pool, tiles=kind.startswith("tiles"))
    want = torch.zeros(T, h, dtype=yt, device="cuda")
    batch.apply([(c.x, want, c.pool)], 0)
    big = torch.full((T + 2, h + 16), float("nan"), dtype=yt, device="cuda")
    got = big[1:-1, 8:8 + h]
    batch.apply([(c.x, got, c.pool)], 0, flags)
    batch.workspace.check()
    assert torch.equal(got, want)
    assert bool(torch.isnan(big[0]).all()) and bool(torch.isnan(big[-1]).all())
    assert bool(torch.isnan(big[:, :8]).all()) and bool(torch.isnan(big[:, 8 + h:]).all())
    bad = c.ids_dev.clone()
    bad[T // 2] = 6                                                # no such adapter: the plan applies nothing
    batch.set_ids(bad, c.pool, tiles=kind.startswith("tiles"))
    got.fill_(float("nan"))
    batch.apply([(c.x, got, c.pool)], 0, flags)
    torch.cuda.synchronize()
    assert bool((got == 0).all())
    assert bool(torch.isnan(big[0]).all()) and bool(torch.isnan(big[:, 8 + h:]).all())


def test_overwrite_clears_the_rows_of_a_segment_that_does_not_fit():
    """A segment whose rank is above what the call's table says is not applied and the call says so: exactly that
    segment's rows are zeros, the others hold their delta."""
    ids = np.array([1, 0, 1, 0, 0], np.int32)
    c = Case(5, 2, 512, 512, np.array([8, 64], np.int32), "fp16", seed=12, ids=ids, n_layers=1)
    want = c.run(0)
    batch = L.LoraBatch(5, 2, 512, 1).set_ids(c.ids_dev, c.pool)
    table = L.adapters_of(c.pool)
    table.r_pool = 8
    y = torch.full((5, 512), 3.0, dtype=torch.float16, device="cuda")
    L.apply([(c.x, y, c.pool)], batch.plan, 0, batch.workspace, _lib.NO_TENSOR | _lib.OVERWRITE, table)
    torch.cuda.synchronize()
    with pytest.raises(L.LoraError) as e:
        batch.workspace.check()
    assert e.value.code == -2
    rows = torch.from_numpy(ids == 0).cuda()
    assert torch.equal(y[rows], want[rows]) and not y[~rows].any()

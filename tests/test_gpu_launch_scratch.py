"""Calls that use no memory of the context, in capture, replay and on two streams: short prefill of f16 rows (the shares of cut tiles are
scratch of the launch) and gated decode pairs of up to 4 rows, on whichever kernel they run.  Results are compared bit for bit with
plain calls."""
import numpy as np
import pytest
import torch

from tests import helpers as H
from tests.gpu_util import ctx

pytestmark = pytest.mark.gpu

# rows, columns, tokens, gated: every tile cut; some cut and some whole; a gated pair of few tiles; decode pairs dealt out by the
# work-list kernel (tiles that fill half the machine)
CALLS = [(300, 4096, 48, False), (43520, 512, 40, False), (200, 2048, 33, True), (4801, 7424, 1, True), (4801, 7424, 4, True)]


def _setup(c, rows, cols, m, gated, seed=200):
    w = [c.prepare_weight(H.Q4_K, H.random_weight(H.Q4_K, rows, cols, seed=seed + i), rows, cols) for i in range(2 if gated else 1)]
    x = torch.from_numpy(np.random.default_rng(seed).standard_normal((m, cols)).astype(np.float32)).to("cuda", torch.float16)
    return w, x


def _call(c, w, x):
    return c.gated_linear(x, *w, out_dtype=torch.float32) if len(w) == 2 else c.linear(x, w[0], out_dtype=torch.float32)


def _fresh():
    from zllm_b200.backend import B200Context

    c = B200Context(0, use_torch_stream=False)
    c.set_option("force_cut_tiles", 1)  # the first three calls' tiles are cut whatever the rule makes of the times
    return c


def _bits(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("rows,cols,m,gated", CALLS)
def test_first_call_of_a_context_can_be_captured_and_replayed_after_any_other(rows, cols, m, gated):
    c, stream = _fresh(), torch.cuda.Stream()
    w, x = _setup(c, rows, cols, m, gated)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        c.set_stream(torch.cuda.current_stream().cuda_stream)
        y = _call(c, w, x)
    c.set_stream(torch.cuda.current_stream().cuda_stream)
    want = _bits(_call(c, w, x))
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(_bits(y), want)
    # calls that make the context's buffers grow, then the graph again
    wide = c.prepare_weight(H.Q4_K, H.random_weight(H.Q4_K, 512, 8192, seed=9), 512, 8192)
    for rows_in in (16, 600, 3000):
        c.linear(torch.zeros((rows_in, 8192), device="cuda"), wide)
    c.linear_batch([(torch.zeros((16, 8192), device="cuda"), wide) for _ in range(8)])  # 8 inputs: more than the first MB of records
    y.zero_()
    for _ in range(3):
        graph.replay()
    c.sync()
    torch.cuda.synchronize()
    assert np.array_equal(_bits(y), want)


@pytest.mark.parametrize("calls", [CALLS[:2], CALLS[3:]])
def test_two_streams_of_one_context(calls):
    c = _fresh()
    jobs = [_setup(c, *call, seed=210 + 4 * i) for i, call in enumerate(calls)]
    streams = [torch.cuda.Stream() for _ in jobs]
    torch.cuda.synchronize()
    c.set_stream(torch.cuda.current_stream().cuda_stream)
    want = [_bits(_call(c, *j)) for j in jobs]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(20):
        for s, j, out in zip(streams, jobs, got):
            with torch.cuda.stream(s):
                c.set_stream(s.cuda_stream)
                out.append(_call(c, *j))
    torch.cuda.synchronize()
    c.sync()
    for out, bits in zip(got, want):
        assert all(np.array_equal(_bits(y), bits) for y in out)


def test_scratch_that_another_shape_has_used():
    """Shapes whose counters and partial sums lie at different places of the same scratch, in turn without a wait."""
    jobs = [_setup(ctx(), *call, seed=230 + 4 * i) for i, call in enumerate(CALLS)]
    want = []
    ctx().set_option("force_cut_tiles", 1)
    try:
        for j in jobs:
            want.append(_bits(_call(ctx(), *j)))
        got = [[_call(ctx(), *j) for j in jobs] for _ in range(10)]
    finally:
        ctx().set_option("force_cut_tiles", 0)
    ctx().sync()
    for outs in got:
        assert all(np.array_equal(_bits(y), bits) for y, bits in zip(outs, want))

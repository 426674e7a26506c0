"""The one-row decode kernels, form by form: which kernel a call runs is read from a captured graph, and every form meets the CPU oracle.

Tolerances are those of the integer-MMA path (tests/test_gpu_gemv.py): 16-bit activations of a 256-column slice, 3e-4; gated results
are products of two such sums, 1e-3; a result in f16 is rounded once more."""
import ctypes
import re

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests import helpers as H
from tests.gpu_util import ctx, dev, host

pytestmark = pytest.mark.gpu

TYPES = [H.Q4_K, H.Q5_K, H.Q6_K, H.Q4_0, H.IQ4_NL, H.Q8_0]
OPTIONS = {"resident": "force_row_resident", "streamed": "force_row_stream", "neither": "disable_row_gemv"}
KERNELS = {"resident": {"gemv_row_kernel"}, "streamed": {"gemv_row_stream_kernel"}}


@pytest.fixture
def force():
    yield lambda form: ctx().set_option(OPTIONS[form], 1)
    ctx().set_option("disable_row_gemv", 0)


DECODE = "gemv_row_stream_kernel|gemv_row_kernel|gemv_i8_kernel|gemv_wl_kernel|wl_quantize_kernel|rmsnorm_kernel"


def launches_of(call, tmp_path, names=DECODE):
    """(name, CTAs, threads) of the kernels of these names that a call launches."""
    call()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    try:
        with torch.cuda.graph(graph):
            ctx().set_stream(torch.cuda.current_stream().cuda_stream)
            call()
    finally:
        ctx().set_stream(torch.cuda.current_stream().cuda_stream)
    dot = tmp_path / "graph.dot"
    assert ctypes.CDLL("libcuda.so.1").cuGraphDebugDotPrint(ctypes.c_void_p(graph.raw_cuda_graph()), str(dot).encode(), 1) == 0
    found = [(name, int(ctas), int(threads)) for name, ctas, threads in re.findall(r"(%s)[^|]*?\\<\\<\\<(\d+),(\d+)," % names, dot.read_text())]
    assert found, "none of the kernels in the graph"
    return found


def kernels_of(call, tmp_path):
    return {name for name, _, _ in launches_of(call, tmp_path)}


def weights(types, rows, cols, seed):
    data = [H.random_weight(t, r, cols, seed=seed + i) for i, (t, r) in enumerate(zip(types, rows))]
    return data, [ctx().prepare_weight(t, d, r, cols) for t, d, r in zip(types, data, rows)]


def fits(form, types, cols, gated):
    """Groups of 16 rows (gated: of gate and of up) beside the records (576 bytes a unit) and the sums of the warps along K: one resident, three or, of
    a pair, two in the ring."""
    unit = {H.Q8_0: 272, H.Q6_K: 224, H.Q5_K: 176}
    units = -(-cols // 256)
    turns = -(-units // 16)
    lanes = -(-units // turns)
    row = max(-(-units * unit.get(t, 144) // 128) * 128 + (32 if t in (H.Q4_K, H.Q5_K) else 64) for t in types)
    groups, sums, limit = (4 if gated else 3, 4, 230400) if form == "streamed" else (2 if gated else 1, 1, 200 * 1024)
    return groups * 16 * row + lanes * turns * 576 + sums * (2 if gated else 1) * lanes * 64 + 128 <= limit


def normed(x, w, eps):
    x = x.astype(np.float64)
    return (x / np.sqrt(np.mean(x * x, axis=-1, keepdims=True) + eps) * w).astype(np.float32)


@pytest.mark.parametrize("tensor_type", TYPES)
@pytest.mark.parametrize("rows,cols,forms", [
    (1, 256, "resident neither"), (17, 768, "resident neither"), (2405, 1024, "resident streamed neither"),  # a unit; three; four, the fewest that are streamed
    (33, 2048, "resident streamed neither"), (513, 4096, "resident streamed neither"),  # eight units: two lanes over the groups; sixteen: one
    (300, 4352, "resident streamed neither"), (40, 16384, "resident streamed neither"),  # two and four turns
])
def test_every_form_meets_the_oracle(force, tmp_path, tensor_type, rows, cols, forms):
    if tensor_type in (H.Q4_0, H.IQ4_NL, H.Q8_0) and cols > 256:
        cols -= 96
    data, w = weights([tensor_type] * 2, [rows] * 2, cols, rows)
    rng = np.random.default_rng(rows + cols)
    x, r = dev(rng.standard_normal((1, cols)).astype(np.float32), torch.bfloat16), dev(rng.standard_normal((1, rows)).astype(np.float32), torch.float16)
    xf = x.float().cpu().numpy()
    plain = orc.linear(tensor_type, data[0], rows, cols, xf) + r.float().cpu().numpy()
    gated = orc.gated_linear(tensor_type, data[0], data[1], rows, cols, xf)
    for form in forms.split():
        force(form)
        for pair, call, want, tol in ((False, lambda: ctx().linear_add(x, w[0], r), plain, 3e-4 + 2 ** -11), (True, lambda: ctx().gated_linear(x, w[0], w[1], out_dtype=torch.float32), gated, 1e-3)):
            ran = kernels_of(call, tmp_path)
            if form == "neither" or not fits(form, [tensor_type], cols, pair):
                assert not ran & {"gemv_row_kernel", "gemv_row_stream_kernel"}
            else:
                assert ran == KERNELS[form]
            assert H.max_rel_error(host(call()), want) <= tol


@pytest.mark.parametrize("shift", [0, 1])  # 1: a row that is not 16-byte aligned
@pytest.mark.parametrize("types,rows,cols", [
    ((H.Q8_0,), (5003,), 1536),                              # six units: two lanes over the groups
    ((H.Q4_K, H.Q4_K, H.Q5_K), (700, 2500, 17), 2048),  # eight; a CTA's range goes on from one projection to the next
    ((H.Q8_0, H.IQ4_NL, H.Q4_0), (900, 33, 2700), 1760), ((H.Q6_K,), (4099,), 3840), ((H.Q4_0, H.IQ4_NL), (300, 1000), 5120),  # two turns
])
@pytest.mark.parametrize("form", ["resident", "streamed", "neither"])
def test_norm_lists_in_every_form(force, tmp_path, form, types, rows, cols, shift):
    eps = 1e-6
    data, ws = weights(types, rows, cols, cols + len(rows))
    rng = np.random.default_rng(cols)
    x = dev((rng.standard_normal(cols + shift) * 3.0).astype(np.float32), torch.float32)[shift:].reshape(1, cols)
    nw = (1.0 + 0.1 * rng.standard_normal(cols)).astype(np.float32)
    weight = dev(nw)
    force(form)
    call = lambda: ctx().rmsnorm_linear_multi(x, weight, eps, ws, out_dtype=torch.float32)
    ran = kernels_of(call, tmp_path)
    assert ran == KERNELS[form] if form != "neither" else not ran & {"gemv_row_kernel", "gemv_row_stream_kernel"}
    xn = normed(x.cpu().numpy(), nw, eps)
    for y, t, d, r in zip(call(), types, data, rows):
        assert H.max_rel_error(host(y), orc.linear(t, d, r, cols, xn)) <= 3e-4


def test_lists_of_both_record_formats_are_not_streamed(force, tmp_path):
    """A CTA's range may hold groups of several projections, and its warps keep the records of one format."""
    data, ws = weights((H.Q4_K, H.Q6_K), (600, 600), 2048, 3)
    x, nw = torch.randn((1, 2048), device="cuda"), torch.rand(2048, device="cuda")
    force("streamed")
    assert "gemv_row_stream_kernel" not in kernels_of(lambda: ctx().rmsnorm_linear_multi(x, nw, 1e-6, ws), tmp_path)


@pytest.mark.parametrize("types,rows,cols,gated,want", [
    ((H.Q4_K,), (512,), 1536, False, "gemv_row_kernel"), ((H.Q4_K, H.Q4_K, H.Q6_K), (1536, 512, 512), 1536, None, "gemv_row_kernel"), ((H.Q4_K,) * 2, (3840,) * 2, 1536, True, "gemv_row_kernel"),
    ((H.Q8_0,), (32768,), 1536, None, "gemv_row_stream_kernel"), ((H.Q8_0,) * 3, (3840,) * 3, 3840, None, "gemv_row_stream_kernel"), ((H.IQ4_NL,) * 2, (15360,) * 2, 3840, True, "gemv_row_stream_kernel"),
])
def test_calls_of_a_decoder_step_take_the_form_they_were_measured_for(tmp_path, types, rows, cols, gated, want):
    ws = weights(types, rows, cols, 1)[1]
    x, nw = torch.randn((1, cols), device="cuda"), torch.rand(cols, device="cuda")
    call = (lambda: ctx().gated_linear(x, *ws)) if gated else (lambda: ctx().linear(x, ws[0])) if gated is False else (lambda: ctx().rmsnorm_linear_multi(x, nw, 1e-6, ws))
    assert kernels_of(call, tmp_path) == {want}


@pytest.mark.parametrize("types,rows,cols", [((H.Q6_K,), (3001,), 2304), ((H.Q4_K, H.Q6_K, H.Q5_K), (3436, 1718, 1718), 2304), ((H.Q6_K,), (4450,), 4608), ((H.Q8_0, H.Q4_K), (2500, 2500), 2048)])
def test_two_ctas_of_an_sm_run_side_by_side(force, tmp_path, types, rows, cols):
    """More CTAs than SMs only where two are resident together.  These kernels take more than 96 registers (Q6_K, several types): four warps per scheduler."""
    ws = weights(types, rows, cols, 1)[1]
    x, nw = torch.randn((1, cols), device="cuda"), torch.rand(cols, device="cuda")
    force("resident")
    for name, ctas, threads in launches_of((lambda: ctx().linear(x, ws[0])) if len(ws) == 1 else lambda: ctx().rmsnorm_linear_multi(x, nw, 1e-6, ws), tmp_path):
        assert name == "gemv_row_kernel"
        assert ctas <= torch.cuda.get_device_properties(0).multi_processor_count or 2 * threads <= 16 * 32


@pytest.mark.parametrize("tensor_type,rows,cols,form", [
    (H.Q4_K, 58000, 256, "norm"), (H.Q4_0, 33709, 512, "norm"), (H.Q4_0, 17408, 512, "plain"), (H.Q5_K, 15939, 2304, "plain"), (H.Q4_K, 6846, 2816, "gated"), (H.Q5_K, 5553, 2304, "gated"), (H.Q4_0, 7200, 3328, "gated"),
])
def test_calls_that_are_faster_elsewhere_are_left_alone(tmp_path, tensor_type, rows, cols, form):
    """Many groups of one or two units, too much for one CTA, a ring for a few groups: 5 to 36 % slower on the one-row kernels."""
    ws = weights((tensor_type,) * 2, (rows,) * (2 if form == "gated" else 1), cols, 1)[1]
    x, nw = torch.randn((1, cols), device="cuda"), torch.rand(cols, device="cuda")
    call = {"plain": lambda: ctx().linear(x, ws[0]), "gated": lambda: ctx().gated_linear(x, *ws), "norm": lambda: ctx().rmsnorm_linear_multi(x, nw, 1e-6, ws)}[form]
    assert not kernels_of(call, tmp_path) & {"gemv_row_kernel", "gemv_row_stream_kernel"}


@pytest.mark.parametrize("types,rows,cols", [((H.Q8_0, H.Q4_0, H.Q4_0), (2000, 9000, 9000), 3328), ((H.Q4_0, H.Q6_K, H.IQ4_NL), (6000, 9000, 3000), 3328), ((H.Q5_K, H.Q4_K, H.Q4_K), (2000, 9000, 9000), 3584)])
def test_a_lists_form_does_not_depend_on_its_order(tmp_path, types, rows, cols):
    ws = weights(types, rows, cols, 1)[1]
    x, nw = torch.randn((1, cols), device="cuda"), torch.rand(cols, device="cuda")
    ran = [kernels_of(lambda: ctx().rmsnorm_linear_multi(x, nw, 1e-6, [ws[i] for i in order]), tmp_path) for order in ((0, 1, 2), (1, 2, 0), (2, 0, 1))]
    assert ran[0] == ran[1] == ran[2]

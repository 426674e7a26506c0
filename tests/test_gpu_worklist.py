"""GPU parity of the work-list decode kernel (``zq_linear_batch`` and the entries built on it) against the CPU
oracle, through the C ABI.

Tolerance: the contract is max_i |a_i - e_i| / max(|e_i|, rms(e)) <= 2e-3 (fp32 accumulation); the integer-MMA
arithmetic (activations as 16-bit integers per 256-column slice, exact integer weights) is held to 3e-4 on top.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests import helpers as H
from tests.gpu_util import ctx, dev, host

pytestmark = pytest.mark.gpu

BOUND = 2e-3
TIGHT = 3e-4


def _check(got, want, tight=TIGHT):
    err = H.max_rel_error(got, want)
    assert err <= BOUND, f"max relative error {err} above the 2e-3 contract"
    assert err <= tight, f"max relative error {err} above the kernel's own {tight}"


def _weight(tensor_type, rows, cols, seed):
    data = H.random_weight(tensor_type, rows, cols, seed=seed)
    return data, ctx().prepare_weight(tensor_type, data, rows, cols)


def test_batch_of_mixed_jobs_matches_cpu_path():
    """Three weight types, every row-count class (1-4, 5-8, 9-16), ragged row counts, odd unit counts, a residual."""
    rng = np.random.default_rng(7)
    specs = [  # (type, rows, cols, m, with residual)
        (H.Q4_K, 200, 1024, 1, False), (H.Q4_K, 130, 768, 4, True), (H.Q4_K, 64, 2560, 3, False), (H.Q4_K, 384, 512, 8, False),
        (H.Q4_K, 257, 1280, 16, True), (H.Q4_0, 7, 96, 1, False), (H.Q4_0, 300, 1056, 2, True), (H.Q4_0, 128, 544, 12, False),
        (H.Q8_0, 64, 1056, 1, False), (H.Q8_0, 2, 32, 4, False), (H.Q8_0, 300, 2560, 6, True), (H.Q4_K, 1000, 256, 1, False),
    ]
    jobs, wants, keep = [], [], []
    for i, (tt, rows, cols, m, res) in enumerate(specs):
        data, w = _weight(tt, rows, cols, 100 + i)
        x = rng.standard_normal((m, cols)).astype(np.float32)
        want = orc.linear(tt, data, rows, cols, x)
        r = None
        if res:
            r = rng.standard_normal((m, rows)).astype(np.float32)
            want = want + r
        jobs.append((dev(x), w, dev(r)) if res else (dev(x), w))
        wants.append(want)
        keep.append(w)
    ys = ctx().linear_batch(jobs)
    for y, want in zip(ys, wants):
        _check(host(y), want)


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q4_0, H.Q8_0, H.IQ4_NL, H.Q5_K, H.Q6_K])
def test_one_tile_cut_across_many_ctas(tensor_type):
    """128 x 17408: one row tile, 34 chunks -> every CTA holds one chunk of the same tile and the last one adds 34 partials."""
    rows, cols = 128, 17408
    data, w = _weight(tensor_type, rows, cols, 5)
    for m in (1, 4, 16):
        x = np.random.default_rng(m).standard_normal((m, cols)).astype(np.float32)
        (y,) = ctx().linear_batch([(dev(x), w)])
        _check(host(y), orc.linear(tensor_type, data, rows, cols, x))


@pytest.mark.parametrize("rows,cols", [(17408, 5120), (5120, 17408)])
def test_full_size_decode_shapes(rows, cols):
    """The two largest matrices of the decode sweep at full size, Q4_K, one and four rows in one batch."""
    data, w = _weight(H.Q4_K, rows, cols, rows)
    x1 = np.random.default_rng(1).standard_normal((1, cols)).astype(np.float32)
    x4 = np.random.default_rng(4).standard_normal((4, cols)).astype(np.float32)
    y1, y4 = ctx().linear_batch([(dev(x1), w), (dev(x4), w)])
    _check(host(y1), orc.linear(H.Q4_K, data, rows, cols, x1))
    _check(host(y4), orc.linear(H.Q4_K, data, rows, cols, x4))
    # the single-call entry on the same weight
    _check(host(ctx().linear(dev(x1), w)), orc.linear(H.Q4_K, data, rows, cols, x1))


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q4_0, H.Q8_0, H.IQ4_NL, H.Q5_K, H.Q6_K])
@pytest.mark.parametrize("m,rows,cols", [(1, 3840, 1536), (1, 100, 512), (4, 192, 1024), (8, 64, 768), (12, 200, 1024)])
def test_gated_jobs_match_cpu_path(tensor_type, m, rows, cols):
    gate, wg = _weight(tensor_type, rows, cols, 21)
    up, wu = _weight(tensor_type, rows, cols, 22)
    x = np.random.default_rng(23).standard_normal((m, cols)).astype(np.float32)
    # a gated job and a plain job in one call
    yg, yp = ctx().linear_batch([(dev(x), wg, wu, "gated"), (dev(x), wu)])
    _check(host(yg), orc.gated_linear(tensor_type, gate, up, rows, cols, x), tight=1e-3)  # silu(g) * u: where u is large and silu(g) small the error of g is weighed by u against the rms of the outputs
    _check(host(yp), orc.linear(tensor_type, up, rows, cols, x))


def test_shared_input_is_quantised_once_and_results_match():
    """dual / triple linear (q, k, v of MiniCPM5: 1536 -> 1536, 512, 512) through the multi-weight entry."""
    cols = 1536
    datas, ws = zip(*[_weight(H.Q4_K, rows, cols, 40 + i) for i, rows in enumerate((1536, 512, 512))])
    x = np.random.default_rng(3).standard_normal((1, cols)).astype(np.float32)
    n0 = ctx().launch_count
    q, k, v = ctx().triple_linear(dev(x), *ws)
    assert ctx().launch_count - n0 == 2, "three projections of one input: one record pass and one decode launch"
    for y, data, rows in zip((q, k, v), datas, (1536, 512, 512)):
        _check(host(y), orc.linear(H.Q4_K, data, rows, cols, x))


def test_results_are_identical_from_run_to_run_and_close_to_single_launches():
    rng = np.random.default_rng(11)
    jobs, keep = [], []
    for i, (rows, cols, m) in enumerate([(3840, 3840, 1), (640, 15360, 4), (2048, 1024, 2)]):
        data, w = _weight(H.Q4_K, rows, cols, 60 + i)
        jobs.append((dev(rng.standard_normal((m, cols)).astype(np.float32)), w))
        keep.append(w)
    a = [host(y).copy() for y in ctx().linear_batch(jobs)]
    b = [host(y).copy() for y in ctx().linear_batch(jobs)]
    for u, v in zip(a, b):
        assert np.array_equal(u.view(np.uint32), v.view(np.uint32))
    ctx().set_option("disable_worklist", 1)
    try:
        c = [host(y).copy() for y in ctx().linear_batch(jobs)]
    finally:
        ctx().set_option("disable_worklist", 0)
    for u, v in zip(a, c):
        assert H.max_rel_error(u, v) <= 1e-5  # same integer arithmetic, different order of the f32 partial sums


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_half_precision_inputs_and_outputs(dtype):
    rows, cols, m = 300, 1024, 3
    data, w = _weight(H.Q4_K, rows, cols, 70)
    x = torch.from_numpy(np.random.default_rng(1).standard_normal((m, cols)).astype(np.float32)).to(dtype)
    (y,) = ctx().linear_batch([(x.cuda(), w)])
    want = orc.linear(H.Q4_K, data, rows, cols, x.float().numpy())
    want = torch.from_numpy(want).to(dtype).float().numpy()  # the output is rounded once to the output dtype
    err = H.max_rel_error(host(y), want)
    assert err <= (1e-3 if dtype == torch.float16 else 8e-3)  # half an ulp of the output type on top of the kernel's error


def test_activation_outlier_inside_a_slice():
    """One activation 1000x the rms of its 256-column slice: the slice is scaled by its maximum, so the small entries keep
    2^-16 of that maximum; the result must stay inside the 2e-3 contract."""
    rows, cols = 512, 2048
    data, w = _weight(H.Q4_K, rows, cols, 80)
    x = np.random.default_rng(2).standard_normal((2, cols)).astype(np.float32)
    x[0, 300] = 1000.0
    x[1, 1500] = -1000.0
    (y,) = ctx().linear_batch([(dev(x), w)])
    err = H.max_rel_error(host(y), orc.linear(H.Q4_K, data, rows, cols, x))
    assert err <= BOUND
    got = host(ctx().linear(dev(x), w))
    assert H.max_rel_error(got, orc.linear(H.Q4_K, data, rows, cols, x)) <= BOUND


def test_unsupported_jobs_fall_back_to_their_own_launches():
    """IQ4_NL and a 40-row job ride in the same call and run as their own launches."""
    rows, cols = 192, 1024
    d1, w1 = _weight(H.IQ4_NL, rows, cols, 90)
    d2, w2 = _weight(H.Q4_K, rows, cols, 91)
    x1 = np.random.default_rng(5).standard_normal((2, cols)).astype(np.float32)
    x2 = np.random.default_rng(6).standard_normal((40, cols)).astype(np.float32)
    y1, y2, y3 = ctx().linear_batch([(dev(x1), w1), (dev(x2), w2), (dev(x1), w2)])
    _check(host(y1), orc.linear(H.IQ4_NL, d1, rows, cols, x1))
    assert H.max_rel_error(host(y2), orc.linear(H.Q4_K, d2, rows, cols, x2)) <= BOUND
    _check(host(y3), orc.linear(H.Q4_K, d2, rows, cols, x1))


def test_argument_errors():
    from zllm_b200 import ffi

    rows, cols = 64, 512
    _, w = _weight(H.Q4_K, rows, cols, 95)
    _, w2 = _weight(H.Q4_K, rows, 256, 96)
    x = dev(np.zeros((1, cols), dtype=np.float32))
    with pytest.raises(ffi.ZqFailure):
        ctx().linear_batch([(x, w, w2, "gated")])  # gate and up differ in shape


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.IQ4_NL])
@pytest.mark.parametrize("m", [1, 5, 16])
def test_gated_pair_whose_tiles_fill_half_the_machine(tensor_type, m):
    """76 tiles of 15 ring items on 148 SMs: dealt out by the work-list kernel (record pass + list), the last tile one row high.
    Against the CPU path by the contract; against the single-matrix kernel, which takes the same activation records and differs
    in the order of its f32 sums only: 2 x 29 terms of one projection are off by 58 x 2^-24 of the sum of their magnitudes, which
    is about sqrt(29) times the result's rms, twice (gate and up): 4e-5."""
    rows, cols = 4801, 7424
    gate, up = H.random_weight(tensor_type, rows, cols, seed=150), H.random_weight(tensor_type, rows, cols, seed=151)
    x = np.random.default_rng(152 + m).standard_normal((m, cols)).astype(np.float32)
    wg, wu = ctx().prepare_weight(tensor_type, gate, rows, cols), ctx().prepare_weight(tensor_type, up, rows, cols)
    before = ctx().launch_count
    got = host(ctx().gated_linear(dev(x), wg, wu))
    assert ctx().launch_count - before == 2
    _check(got, orc.gated_linear(tensor_type, gate, up, rows, cols, x), tight=BOUND)
    ctx().set_option("disable_worklist", 1)
    try:
        alone = host(ctx().gated_linear(dev(x), wg, wu))
    finally:
        ctx().set_option("disable_worklist", 0)
    assert H.max_rel_error(got, alone) <= 4e-5


def test_first_gated_call_of_a_context_can_be_captured():
    """The gated pair that goes to the work-list kernel finds its record buffer in place: no allocation under capture."""
    from zllm_b200.backend import B200Context

    rows, cols = 4801, 7424
    data = H.random_weight(H.Q4_K, rows, cols, seed=170)
    c = B200Context(0, use_torch_stream=False)
    stream = torch.cuda.Stream()
    w = c.prepare_weight(H.Q4_K, data, rows, cols)
    x = dev(np.random.default_rng(171).standard_normal((4, cols)).astype(np.float32))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        c.set_stream(torch.cuda.current_stream().cuda_stream)
        y = c.gated_linear(x, w, w)
    graph.replay()
    torch.cuda.synchronize()
    _check(host(y), orc.gated_linear(H.Q4_K, data, data, rows, cols, x.cpu().numpy()), tight=BOUND)


@pytest.mark.parametrize("pinned", [True, False])
def test_bracket_that_sends_its_layers_out_in_several_batches(pinned):
    """16 rows: the fourth input takes longer to arrive than the layers before it to run, so this list is sent in parts; an input read
    before and after a part goes out, inputs that arrive while one runs.  Twice, with other inputs."""
    m = 16
    shapes = [(2048, 8192, 0), (1024, 16400, 1), (2048, 300, 0), (17408, 640, 2), (1024, 72, 1)]  # columns, rows, input
    weights = [(_weight(H.Q4_0, rows, cols, 180 + i), cols, rows, k) for i, (cols, rows, k) in enumerate(shapes)]
    for seed in (190, 191):
        rng = np.random.default_rng(seed)

        def buf(shape):
            t = torch.zeros(shape)
            return (t.pin_memory() if pinned else t)

        xs = {k: buf((m, cols)) for _, cols, _, k in weights}
        for t in xs.values():
            t.copy_(torch.from_numpy(rng.standard_normal(tuple(t.shape)).astype(np.float32)))
        ys = [buf((m, rows)) for _, _, rows, _ in weights]
        ctx().linear_host_batch([(xs[k].numpy(), w, y.numpy()) for ((_, w), _, _, k), y in zip(weights, ys)])
        for ((data, _), cols, rows, k), y in zip(weights, ys):
            _check(y.numpy(), orc.linear(H.Q4_0, data, rows, cols, xs[k].numpy()))


@pytest.mark.parametrize("pinned", [True, False])
def test_bracket_collects_layers_while_the_gpu_is_busy(pinned):
    """Results of 1.1 MB each, one small input: nothing that a layer waits for, so the layers collect while those before them run; the same
    list runs as the same launches every time, and its results do not depend on what ran before."""
    m, rows, cols = 16, 17408, 512
    made = [_weight(H.Q4_0, rows, cols, 300 + i) for i in range(8)]

    def buf(shape):
        t = torch.zeros(shape)
        return t.pin_memory() if pinned else t

    x = buf((m, cols))
    x.copy_(torch.from_numpy(np.random.default_rng(301).standard_normal((m, cols)).astype(np.float32)))
    ys = [buf((m, rows)) for _ in made]
    counts, bits = [], []
    for _ in range(3):
        before = ctx().launch_count
        ctx().linear_host_batch([(x.numpy(), w, y.numpy()) for (_, w), y in zip(made, ys)])
        counts.append(ctx().launch_count - before)
        bits.append([y.numpy().view(np.uint32).copy() for y in ys])
    assert counts == [counts[0]] * 3 and counts[0] <= 8  # 16: a record pass and a launch for every layer
    assert all(np.array_equal(a, b) for run in bits[1:] for a, b in zip(run, bits[0]))
    for (data, _), y in zip(made, ys):
        _check(y.numpy(), orc.linear(H.Q4_0, data, rows, cols, x.numpy()))


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q8_0, H.Q6_K])
@pytest.mark.parametrize("gated,m,jobs,finisher", [(False, 5, 8, True), (False, 8, 8, True), (False, 8, 5, False), (True, 5, 6, True), (True, 7, 6, True), (True, 8, 3, False)])
def test_lists_of_5_to_8_rows_on_both_sides_of_the_finisher_rule(tensor_type, gated, m, jobs, finisher):
    """71 (gated 141) tiles of 3 ring items per job, ranges that cut them: long lists leave cut tiles to the finisher warp, short ones to
    the consumers.  Against the CPU path, and against the jobs run alone on the single-matrix kernel (same records, other order of the
    f32 sums: 2 x 11 terms, the bound of the gated pair above with room)."""
    rows, cols = 9000, 1536
    per_cta = jobs * (3 * 141 if gated else 3 * 71) // ctx().sm_count
    assert (per_cta - 3 >= 2 * m - (0 if gated else 8)) == finisher
    data = [H.random_weight(tensor_type, rows, cols, seed=310 + i) for i in range(2)]
    ws = [ctx().prepare_weight(tensor_type, d, rows, cols) for d in data]
    xs = [dev(np.random.default_rng(320 + i).standard_normal((m, cols)).astype(np.float32)) for i in range(jobs)]
    listed = [(x, ws[0], ws[1], "gated") if gated else (x, ws[i % 2]) for i, x in enumerate(xs)]
    got = [host(y) for y in ctx().linear_batch(listed)]
    ctx().set_option("disable_worklist", 1)
    try:
        alone = [host(y) for y in ctx().linear_batch(listed)]
    finally:
        ctx().set_option("disable_worklist", 0)
    for a, b in zip(got, alone):
        assert H.max_rel_error(a, b) <= 4e-5
    for i in (0, jobs - 1):
        x = xs[i].cpu().numpy()
        want = orc.gated_linear(tensor_type, data[0], data[1], rows, cols, x) if gated else orc.linear(tensor_type, data[i % 2], rows, cols, x)
        _check(got[i], want, tight=BOUND)


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q5_K, H.Q6_K, H.Q4_0, H.IQ4_NL, H.Q8_0])
@pytest.mark.parametrize("specs,fits", [
    ([(200, 1536, 1), (130, 256, 4), (257, 2560, 3)], True),                  # odd units, one unit, ragged rows
    ([(3840, 3840, 1), (3840, 512, 1), (15000, 1024, 2)], True),              # ranges that hold parts of two inputs
    ([(640, 17408, 1), (300, 16384, 4), (129, 8192, 4)], True),               # long rows, of which a range needs a few units
    ([(2000, 4352, 2), (1000, 2048, 1)], True),                               # ranges of two items that go from a row's last chunk (one unit) to its first
    ([(5120, 8192, 2), (3000, 8448, 2), (5120, 8192, 2)], True),              # ranges of 12 items: parts of a row that go round, a shorter ring
    ([(5120, 8192, 4), (3000, 8448, 4), (5120, 8192, 4), (5120, 8192, 4)], False),  # more records than are worth it: the record pass
])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_records_in_shared_memory_give_the_bits_of_the_record_pass(tensor_type, specs, fits, dtype):
    """Lists of up to 4 rows quantise their inputs inside the decode kernel.  A result that lies over an input (here: the first job's over the
    last one's) sends the same list through the record pass: same ranges, same order of every sum."""
    from zllm_b200 import ffi

    rng = np.random.default_rng(400 + len(specs) + specs[0][1])
    made = {}
    for rows, cols, _ in specs:
        if (rows, cols) not in made:
            made[rows, cols] = ctx().prepare_weight(tensor_type, H.random_weight(tensor_type, rows, cols, seed=401 + len(made)), rows, cols)
    ws = [made[rows, cols] for rows, cols, _ in specs]
    xs = [dev(rng.standard_normal((m, cols)).astype(np.float32), dtype) for _, cols, m in specs]

    def run(over):
        jobs = (ffi.ZqLinearJob * len(specs))()
        ys = [torch.zeros(m * rows, device="cuda") for rows, _, m in specs]
        inputs = [x.clone() for x in xs]
        for j, (rows, cols, m), w, x, y in zip(jobs, specs, ws, inputs, ys):
            j.w, j.dev_x, j.m, j.dev_y = w.handle, x.data_ptr(), m, y.data_ptr()
        if over:  # the last input inside the first result's buffer: read before anything is written
            need = xs[-1].numel() * xs[-1].element_size()
            buf = torch.zeros(max(specs[0][0] * specs[0][2] * 4, need), dtype=torch.uint8, device="cuda")
            buf[:need] = xs[-1].reshape(-1).view(torch.uint8)
            jobs[len(specs) - 1].dev_x = jobs[0].dev_y = buf.data_ptr()
            ys[0] = buf[: specs[0][0] * specs[0][2] * 4].view(torch.float32)
        before = ctx().launch_count
        code = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[dtype]
        ffi.call("zq_linear_batch", ctx().handle, jobs, len(specs), code, 0)
        ctx().sync()
        return [host(y).copy() for y in ys], ctx().launch_count - before

    (inside, n_inside), (passed, n_passed) = run(False), run(True)
    assert n_passed == 2 and n_inside == (1 if fits else 2)
    for a, b in zip(inside, passed):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("types,m", [((H.Q4_K, H.Q6_K), 1), ((H.Q4_K, H.Q6_K), 4), ((H.Q8_0, H.Q5_K, H.IQ4_NL), 1), ((H.Q4_0, H.Q8_0, H.Q4_K, H.Q5_K, H.Q6_K, H.IQ4_NL), 1)])
def test_lists_of_several_types_in_one_launch(types, m):
    rng = np.random.default_rng(430 + m)
    made = [(t, rows, cols, *_weight(t, rows, cols, 431 + i)) for i, (t, rows, cols) in enumerate((t, 130 + 257 * i, 256 * (1 + 3 * (i % 3))) for i, t in enumerate(types))]
    xs = [rng.standard_normal((m, cols)).astype(np.float32) for _, _, cols, _, _ in made]
    before = ctx().launch_count
    ys = ctx().linear_batch([(dev(x), w) for x, (*_, w) in zip(xs, made)])
    assert ctx().launch_count - before == 1
    for y, x, (t, rows, cols, data, _) in zip(ys, xs, made):
        _check(host(y), orc.linear(t, data, rows, cols, x))


@pytest.mark.parametrize("types", [(H.Q4_K,), (H.Q4_K, H.Q8_0), (H.Q8_0, H.Q6_K, H.Q5_K)])
def test_norm_inside_the_decode_kernel_and_before_it(types):
    """One row: norm and projections in one launch, the bits of the norm kernel in front (which a second row brings back)."""
    cols, rows = 3840, 300
    ws = [_weight(t, rows + i, cols, 440 + i)[1] for i, t in enumerate(types)]
    x = dev(np.random.default_rng(441).standard_normal((1, cols)).astype(np.float32) * 2.0)
    nw = dev((1.0 + 0.1 * np.random.default_rng(442).standard_normal(cols)).astype(np.float32))
    before = ctx().launch_count
    one = [host(y) for y in ctx().rmsnorm_linear_multi(x, nw, 1e-5, ws)]
    assert ctx().launch_count - before == 1
    two = [host(y) for y in ctx().rmsnorm_linear_multi(torch.cat([x, x]), nw, 1e-5, ws)]
    for a, b in zip(one, two):
        if len(types) == 1:
            assert np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32))
        assert H.max_rel_error(a, b[:1]) <= 1e-5  # two types share a launch in one case: other ranges, other order of the f32 sums


@pytest.mark.parametrize("offset", [0, 2560])  # the row at the front of the result's buffer, and inside it
def test_gated_row_under_its_own_result_keeps_the_record_pass(offset):
    """One row, its result over it: the records are made before anything is stored (two launches), not by CTAs that store side by side (one)."""
    from zllm_b200 import ffi

    rows, cols = 10240, 5120
    data = [H.random_weight(H.Q4_K, rows, cols, seed=s) for s in (1, 2)]
    w = [ctx().prepare_weight(H.Q4_K, d, rows, cols) for d in data]
    x = torch.randn((1, cols), generator=torch.Generator().manual_seed(5)).cuda()
    run = lambda src, dst: ffi.call("zq_gated_silu", ctx().handle, w[0].handle, w[1].handle, src.data_ptr(), 0, 1, dst.data_ptr(), 0)
    apart = torch.empty((1, rows), device="cuda")
    before = ctx().launch_count
    run(x, apart)
    assert ctx().launch_count - before == 1
    buffer = torch.zeros((1, rows), device="cuda")
    under = buffer[:, offset:offset + cols]
    under.copy_(x)
    before = ctx().launch_count
    run(under, buffer)
    assert ctx().launch_count - before == 2
    want = orc.gated_linear(H.Q4_K, data[0], data[1], rows, cols, x.cpu().numpy())
    assert H.max_rel_error(host(buffer), want) <= 1e-3 and H.max_rel_error(host(apart), want) <= 1e-3  # products of two sums

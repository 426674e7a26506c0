"""GPU parity of the prefill GEMM (tcgen05 path, more than 16 activation rows) against the CPU oracle.

Tolerance: max_i |a_i - e_i| / max(|e_i|, rms(e)) <= 2e-3.  The tensor-core path rounds dequantised weights and
activations to f16 once (2^-12 relative each) and accumulates in f32; the oracle consumes the same activation
values the device consumes (bf16/f16 inputs are exact in f16).
"""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests import helpers as H
from tests.gpu_util import ctx, dev, host

pytestmark = pytest.mark.gpu
BOUND = 2e-3


@pytest.fixture(autouse=True, params=["fused", "operand_pass"])
def gemm_variant(request):
    """Every decode type runs on the kernel that dequantises inside the GEMM and on the separate f16 operand pass + plain GEMM, and every
    case on both.  Their operands are the same bits; results are where both deal their tiles out alike."""
    ctx().set_option("disable_fused_gemm", 1 if request.param == "operand_pass" else 0)
    ctx().set_option("force_fused_gemm", 1 if request.param == "fused" else 0)
    yield request.param
    ctx().set_option("disable_fused_gemm", 0)
    ctx().set_option("force_fused_gemm", 0)


@pytest.fixture
def cut_tiles():
    """Tiles are cut along K wherever they can be, whatever the rule makes of the times."""
    ctx().set_option("force_cut_tiles", 1)
    yield
    ctx().set_option("force_cut_tiles", 0)


def test_fused_and_operand_pass_kernels_agree_bit_for_bit(gemm_variant):
    if gemm_variant == "operand_pass":
        pytest.skip("compares a fused variant with the operand pass in one go")
    rows, cols, m = 300, 1024, 530
    data = H.random_weight(H.Q4_K, rows, cols, seed=77)
    x = dev(np.random.default_rng(78).standard_normal((m, cols)).astype(np.float32), torch.bfloat16)
    w = ctx().prepare_weight(H.Q4_K, data, rows, cols)
    a = host(ctx().linear(x, w, out_dtype=torch.float32)).copy()
    ctx().set_option("force_fused_gemm", 0)
    ctx().set_option("disable_fused_gemm", 1)
    b = host(ctx().linear(x, w, out_dtype=torch.float32))
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q4_0, H.Q8_0, H.IQ4_NL])
@pytest.mark.parametrize("m,rows,cols", [(17, 200, 1024), (64, 128, 256), (300, 384, 2048), (512, 130, 512)])
def test_prefill_linear_matches_cpu_matmul(tensor_type, m, rows, cols):
    data = H.random_weight(tensor_type, rows, cols, seed=3 * m + rows)
    x = np.random.default_rng(m).standard_normal((m, cols)).astype(np.float32)
    x16 = dev(x, torch.bfloat16)
    w = ctx().prepare_weight(tensor_type, data, rows, cols)
    got = host(ctx().linear(x16, w, out_dtype=torch.float32))
    want = orc.linear(tensor_type, data, rows, cols, x16.float().cpu().numpy())
    assert H.max_rel_error(got, want) <= BOUND


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q5_K, H.Q6_K, H.Q4_0, H.IQ4_NL, H.Q8_0])
@pytest.mark.parametrize("m,rows,cols,gated", [
    (17, 1, 256, False), (32, 300, 512, True), (64, 19300, 1280, False),  # four units of tokens in the ring; pairs that walk two tiles on an odd number of units
    (65, 9800, 768, True), (96, 130, 2816, False), (128, 19300, 1536, False), (128, 9800, 1280, True), (129, 300, 1280, False),  # two units; past the largest short tile
])
def test_short_tiles_agree_with_the_operand_pass_bit_for_bit(gemm_variant, tensor_type, m, rows, cols, gated):
    """The weight operand in tensor memory is the operand pass's, k for k: whole tiles have the same bits."""
    if gemm_variant == "operand_pass":
        pytest.skip("compares a fused variant with the operand pass in one go")
    if tensor_type in (H.Q4_0, H.IQ4_NL, H.Q8_0):
        cols -= 96
    g = torch.Generator(device="cuda").manual_seed(m + rows)
    make = lambda: ctx().prepare_weight(tensor_type, H.random_weight(tensor_type, rows, cols, seed=int(torch.randint(0, 1000, (1,), generator=g, device="cuda"))), rows, cols)
    w = [make() for _ in range(2 if gated else 1)]
    x = torch.randn((m, cols), generator=g, device="cuda").to(torch.float16)
    run = lambda: ctx().gated_linear(x, *w, out_dtype=torch.float32) if gated else ctx().linear(x, w[0], out_dtype=torch.float32)
    ctx().set_option("disable_cut_tiles", 1)
    try:
        a = run()
        ctx().set_option("force_fused_gemm", 0)
        ctx().set_option("disable_fused_gemm", 1)
        b = run()
    finally:
        ctx().set_option("disable_cut_tiles", 0)
    assert torch.isfinite(a).all()
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))


def test_prefill_reference_generator_case():
    """src/kernel/cuda/linear.rs:2176-2206 shape (M = 9 runs the decode kernel; M = 33 the tensor-core path) with
    the reference's own device gate 0.05 + 0.002*|e| as an outer bound."""
    rows, cols, m = 2, 256, 33
    packed = H.reference_packed_blocks(12, rows)
    idx = np.arange(m * cols, dtype=np.int64)
    x = (((idx * 17 % 101).astype(np.float32) - 50.0) / 64.0).reshape(m, cols)
    w = ctx().prepare_weight(12, packed, rows, cols)
    got = host(ctx().linear(dev(x, torch.float16), w, out_dtype=torch.float32))
    want = orc.linear(12, packed, rows, cols, x)
    assert np.all(np.abs(got - want) <= 0.05 + 0.002 * np.abs(want))
    assert H.max_rel_error(got, want) <= BOUND


@pytest.mark.parametrize("y_dtype", [torch.bfloat16, torch.float16])
def test_prefill_output_dtypes_and_residual(y_dtype):
    rows, cols, m = 256, 768, 100
    data = H.random_weight(H.Q4_K, rows, cols, seed=5)
    x = dev(np.random.default_rng(6).standard_normal((m, cols)).astype(np.float32), torch.bfloat16)
    r = dev(np.random.default_rng(7).standard_normal((m, rows)).astype(np.float32), y_dtype)
    w = ctx().prepare_weight(H.Q4_K, data, rows, cols)
    got = host(ctx().linear_add(x, w, r))
    want = orc.linear(H.Q4_K, data, rows, cols, x.float().cpu().numpy()) + r.float().cpu().numpy()
    tol = BOUND + (2 ** -8 if y_dtype == torch.bfloat16 else 2 ** -11)  # compute bound + rounding of the stored dtype
    assert H.max_rel_error(got, want) <= tol


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q4_0])
def test_prefill_gated_matches_cpu_path(tensor_type):
    """src/kernel/cuda/linear.rs:2317-2355 (gated Q4_K prefill, M = 9 there; 40 here to reach the tensor-core path)."""
    rows, cols, m = 320, 512, 40
    gate, up = H.random_weight(tensor_type, rows, cols, seed=8), H.random_weight(tensor_type, rows, cols, seed=9)
    x = dev(np.random.default_rng(10).standard_normal((m, cols)).astype(np.float32), torch.bfloat16)
    wg, wu = ctx().prepare_weight(tensor_type, gate, rows, cols), ctx().prepare_weight(tensor_type, up, rows, cols)
    got = host(ctx().gated_linear(x, wg, wu, out_dtype=torch.float32))
    want = orc.gated_linear(tensor_type, gate, up, rows, cols, x.float().cpu().numpy())
    assert H.max_rel_error(got, want) <= BOUND


def test_prefill_full_width_slice():
    """One 128-row x 256-token tile of the 5120 -> 17408 prefill shape at full K, checked on a seeded subsample."""
    rows, cols, m = 128, 5120, 256
    data = H.random_weight(H.Q4_K, rows, cols, seed=11)
    x = dev(np.random.default_rng(12).standard_normal((m, cols)).astype(np.float32), torch.bfloat16)
    w = ctx().prepare_weight(H.Q4_K, data, rows, cols)
    got = host(ctx().linear(x, w, out_dtype=torch.float32))
    sel = np.random.default_rng(13).choice(m, size=24, replace=False)
    want = orc.linear(H.Q4_K, data, rows, cols, x.float().cpu().numpy()[sel])
    assert H.max_rel_error(got[sel], want) <= BOUND


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q5_K, H.Q6_K, H.Q4_0, H.IQ4_NL, H.Q8_0])
@pytest.mark.parametrize("m,rows,cols", [
    (17, 1, 256), (33, 129, 1280), (255, 255, 512), (257, 257, 768),  # edges of 32-token groups, 128 / 256-row tiles; shares of one tile
    (40, 25600, 512),   # 100 tiles: every tile cut along K
    (40, 43520, 512),   # 170 tiles: 96 of them cut, 74 whole
])
def test_prefill_tiles_and_shares(tensor_type, m, rows, cols, cut_tiles):
    """Edges of the pair's tile (32 tokens, 128 and 256 rows) and the three ways tiles are dealt (whole, cut, both), with a
    residual; block-32 types on columns that end inside a k-block.  Bound as above: both operands are rounded to f16 once."""
    if tensor_type in (H.Q4_0, H.IQ4_NL, H.Q8_0):
        cols -= 160
    # weights inside the f16 operand's range (|w| <= 65504): arbitrary scale bits give weights of 1e8 and an infinite operand
    data = H.random_weight(tensor_type, rows, cols, seed=m + rows)
    x = dev(np.random.default_rng(m).standard_normal((m, cols)).astype(np.float32), torch.bfloat16)
    r = np.random.default_rng(m + 1).standard_normal((m, rows)).astype(np.float32)
    w = ctx().prepare_weight(tensor_type, data, rows, cols)
    got = host(ctx().linear(x, w, out_dtype=torch.float32, residual=dev(r)))
    sel = np.unique(np.concatenate([np.random.default_rng(m + 2).choice(m, size=min(m, 9), replace=False), [0, m - 1]]))
    want = orc.linear(tensor_type, data, rows, cols, x.float().cpu().numpy()[sel]) + r[sel]
    assert H.max_rel_error(got[sel], want) <= BOUND


@pytest.mark.parametrize("tensor_type,m,rows,cols,gated,dtype", [
    (H.Q4_K, 40, 2100, 3072, False, torch.float32), (H.Q5_K, 40, 2100, 3072, False, torch.bfloat16), (H.Q6_K, 40, 2100, 3072, False, torch.float16),
    (H.Q4_0, 40, 2100, 3072, False, torch.float32), (H.IQ4_NL, 40, 2100, 3072, False, torch.bfloat16), (H.Q8_0, 40, 2100, 3072, False, torch.float16),
    (H.Q4_K, 300, 333, 8192, False, torch.float16),   # two token tiles, rows that are no multiple of 4
    (H.Q4_K, 256, 511, 8192, False, torch.float32),   # whole 256-token tiles
    (H.Q4_K, 40, 43520, 3072, False, torch.float32),  # 170 tiles: 96 of them cut, 74 whole
    (H.Q4_K, 70, 700, 3072, True, torch.float32), (H.Q8_0, 256, 77, 8192, True, torch.float16), (H.IQ4_NL, 33, 1030, 4096, True, torch.bfloat16),
    (H.Q6_K, 290, 2001, 2048, False, torch.float32), (H.Q4_K, 610, 900, 4096, False, torch.float32), (H.Q5_K, 280, 700, 2048, True, torch.float32),  # wide where dequantised inside
])
def test_prefill_cut_tiles(tensor_type, m, rows, cols, gated, dtype, cut_tiles):
    """Long rows and few tiles: cut along K and added up at the end, with residual, every output type, ragged rows and tokens.
    Bounds as in the tests around this one, plus the rounding of a 16-bit output (2^-9 bf16, 2^-12 f16).  That tiles were cut shows in
    the last bits of f32 results, whose sums are in another order than those of whole tiles."""
    ws = [H.random_weight(tensor_type, rows, cols, seed=m + rows + i) for i in range(2 if gated else 1)]
    x = dev(np.random.default_rng(m).standard_normal((m, cols)).astype(np.float32), torch.float16)
    wd = [ctx().prepare_weight(tensor_type, w, rows, cols) for w in ws]
    sel = np.unique(np.concatenate([np.random.default_rng(m + 2).choice(m, size=min(m, 7), replace=False), [0, m - 1]]))
    xs = x.float().cpu().numpy()[sel]
    rounding = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    r = None if gated else dev(np.random.default_rng(m + 1).standard_normal((m, rows)).astype(np.float32), dtype)

    def run():
        return host((ctx().gated_linear(x, *wd, out_dtype=dtype) if gated else ctx().linear(x, wd[0], out_dtype=dtype, residual=r)).float())

    ctx().set_option("force_wide_tiles", 1)
    try:
        got = run()
        if dtype == torch.float32:
            ctx().set_option("disable_cut_tiles", 1)
            whole = run()
            assert not np.array_equal(got, whole) and H.max_rel_error(got, whole) <= 1e-4
    finally:
        ctx().set_option("force_wide_tiles", 0)
    if gated:
        assert H.max_rel_error(got[sel], orc.gated_linear(tensor_type, *ws, rows, cols, xs)) <= 2.1 * BOUND + rounding
        return
    want = orc.linear(tensor_type, ws[0], rows, cols, xs) + r.float().cpu().numpy()[sel]
    assert H.max_rel_error(got[sel], want) <= BOUND + rounding


@pytest.mark.parametrize("tensor_type,rows,m,gated,dtype", [
    (H.Q4_K, 17300, 257, False, torch.float32),   # one wide tile of 9 chunks, one pair per tile; ragged rows
    (H.Q6_K, 17408, 320, False, torch.bfloat16),  # full width, 10 chunks
    (H.Q4_K, 17408, 900, False, torch.float16),   # three wide tiles per pair: their accumulators overlap
    (H.Q8_0, 11008, 830, False, torch.float32),   # the last of three tiles is not wide
    (H.Q5_K, 17408, 300, False, torch.float16), (H.IQ4_NL, 17408, 289, False, torch.float32), (H.Q4_0, 17408, 290, False, torch.float32),
    (H.IQ4_NL, 3840, 560, True, torch.float16),   # gated
])
def test_prefill_wide_tiles(tensor_type, rows, m, gated, dtype, gemm_variant):
    """Tiles of 257 to 320 tokens give the bits of the operand pass, whose tiles end at 256 (whole tiles on both sides: no sum is split)."""
    if gemm_variant == "operand_pass":
        pytest.skip("compares the two in one go")
    cols = 512
    ws = [ctx().prepare_weight(tensor_type, H.random_weight(tensor_type, rows, cols, seed=500 + i), rows, cols) for i in range(2 if gated else 1)]
    x = dev(np.random.default_rng(501).standard_normal((m, cols)).astype(np.float32), torch.float16)
    r = None if gated else dev(np.random.default_rng(502).standard_normal((m, rows)).astype(np.float32), dtype)

    def run():
        return (ctx().gated_linear(x, *ws, out_dtype=dtype) if gated else ctx().linear(x, ws[0], out_dtype=dtype, residual=r)).clone()

    a = run()
    ctx().set_option("force_fused_gemm", 0)
    ctx().set_option("disable_fused_gemm", 1)
    assert torch.equal(a, run())


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q8_0, H.Q6_K])
@pytest.mark.parametrize("m,rows,cols", [(31, 63, 512), (260, 130, 1024)])
def test_prefill_gated_edges(tensor_type, m, rows, cols):
    """64 gate and 64 up rows share a tile: ragged row counts, one and two token tiles, shares of a tile.
    Bound: the output is a product of two projections, each within BOUND of its own scale, through a SiLU of slope at most
    1.1: |d(silu(g) u)| <= 1.1 |dg| |u| + |silu(g)| |du|, i.e. 2.1 BOUND."""
    gate, up = H.random_weight(tensor_type, rows, cols, seed=rows), H.random_weight(tensor_type, rows, cols, seed=rows + 1)
    x = dev(np.random.default_rng(rows).standard_normal((m, cols)).astype(np.float32), torch.float16)
    wg, wu = ctx().prepare_weight(tensor_type, gate, rows, cols), ctx().prepare_weight(tensor_type, up, rows, cols)
    got = host(ctx().gated_linear(x, wg, wu, out_dtype=torch.float32))
    sel = [0, 1, m // 2, m - 1]
    want = orc.gated_linear(tensor_type, gate, up, rows, cols, x.float().cpu().numpy()[sel])
    assert H.max_rel_error(got[sel], want) <= 2.1 * BOUND


@pytest.mark.parametrize("m", [17, 48, 300])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_projections_that_feed_each_other_wait_for_each_other(m, dtype):
    """A GEMM is set up under the kernel before it (operand conversion or another GEMM): a chain enqueued at once gives the bits of
    the same chain with a wait behind every call."""
    cols = 1024
    ws = [ctx().prepare_weight(t, H.random_weight(t, cols, cols, seed=160 + i), cols, cols) for i, t in enumerate((H.Q4_K, H.Q8_0, H.IQ4_NL, H.Q6_K))]
    x0 = torch.from_numpy(np.random.default_rng(161).standard_normal((m, cols)).astype(np.float32)).to("cuda", dtype)

    def chain(wait):
        x, outs = x0, []
        for i in range(8):
            y = ctx().linear(x, ws[i % 4], residual=x)
            if wait:
                ctx().sync()
            x = (y * 0.5).to(dtype)
            outs.append(ctx().gated_linear(x, ws[i % 4], ws[i % 4], out_dtype=torch.float32))
        ctx().sync()
        return [o.cpu().numpy() for o in outs]

    want = chain(True)
    for _ in range(3):
        for a, b in zip(chain(False), want):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q5_K, H.Q6_K, H.Q4_0, H.IQ4_NL, H.Q8_0])
def test_operand_is_the_dequantised_value_rounded_once(tensor_type):
    """Rows of the identity as activations (exact in f16, one non-zero product per sum) read the weight operand back bit for bit:
    the codec's f32 value rounded once to f16, for scale and minimum of any ratio, down to values that nearly cancel."""
    rows, cols = 300, 512
    e, b = orc.BLOCK[tensor_type]
    data = H.random_bytes_weight(tensor_type, rows, cols, seed=17).reshape(-1, b)
    rng = np.random.default_rng(18)
    exponent = rng.integers(-14, -4, size=len(data))
    scales = [np.ldexp(1.0 + rng.random(len(data)), exponent).astype(np.float16)]
    if len(H.SCALE_OFFSETS[tensor_type]) == 2:  # minimum: 2^-9 .. 2^15 times the scale, as far as f16 goes
        scales.append(np.ldexp(1.0 + rng.random(len(data)), np.minimum(exponent + rng.integers(-9, 16, size=len(data)), 8)).astype(np.float16))
    for off, v in zip(H.SCALE_OFFSETS[tensor_type], scales):
        data[:, off:off + 2] = v.view(np.uint8).reshape(-1, 2)
    data = data.reshape(-1)
    want = orc.dequantize(tensor_type, data, rows * cols).reshape(rows, cols).astype(np.float16)
    w = ctx().prepare_weight(tensor_type, data, rows, cols)
    got = host(ctx().linear(torch.eye(cols, device="cuda", dtype=torch.float16), w, out_dtype=torch.float32)).T
    assert np.array_equal(got, want.astype(np.float32))


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q5_K])
def test_k_quant_operand_at_the_edges_of_the_scale_range(tensor_type):
    """Scale and minimum that are zero, negative, subnormal f16 or as large as the operand's range allows (31 * 63 * 32 < 65504): the operand is
    the codec's value rounded once, bit for bit (a zero's sign does not survive the sum)."""
    rows, cols = 96, 256
    e, b = orc.BLOCK[tensor_type]
    data = H.random_bytes_weight(tensor_type, rows, cols, seed=19).reshape(-1, b)
    edges = np.array([0.0, -0.0, 2.0 ** -24, -3 * 2.0 ** -24, 1023 * 2.0 ** -24, 2.0 ** -14, 0.3, -0.3, 31.0, -32.0], np.float16)
    rng = np.random.default_rng(20)
    for off in H.SCALE_OFFSETS[tensor_type]:
        data[:, off:off + 2] = rng.choice(edges, size=len(data)).view(np.uint8).reshape(-1, 2)
    data = data.reshape(-1)
    want = orc.dequantize(tensor_type, data, rows * cols).reshape(rows, cols).astype(np.float16)
    w = ctx().prepare_weight(tensor_type, data, rows, cols)
    got = host(ctx().linear(torch.eye(cols, device="cuda", dtype=torch.float16), w, out_dtype=torch.float32)).T
    assert np.isfinite(want).all() and np.array_equal(got, want.astype(np.float32))


@pytest.mark.parametrize("tensor_type", [H.Q4_K, H.Q5_K, H.Q6_K, H.Q4_0, H.IQ4_NL, H.Q8_0])
@pytest.mark.parametrize("gated", [False, True])
def test_both_operand_forms_agree_bit_for_bit_for_every_type(tensor_type, gated, gemm_variant):
    if gemm_variant == "operand_pass":
        pytest.skip("compares a fused variant with the operand pass in one go")
    rows, m = 300, 530
    cols = 1024 if tensor_type in (H.Q4_K, H.Q5_K, H.Q6_K) else 1024 - 96
    ws = [ctx().prepare_weight(tensor_type, H.random_weight(tensor_type, rows, cols, seed=177 + i), rows, cols) for i in range(2)]
    x = dev(np.random.default_rng(178).standard_normal((m, cols)).astype(np.float32), torch.bfloat16)

    def run():
        return host(ctx().gated_linear(x, *ws, out_dtype=torch.float32) if gated else ctx().linear(x, ws[0], out_dtype=torch.float32)).copy()

    a = run()
    ctx().set_option("force_fused_gemm", 0)
    ctx().set_option("disable_fused_gemm", 1)
    assert np.array_equal(a.view(np.uint32), run().view(np.uint32))


@pytest.mark.parametrize("m", [17, 48, 300, 1100])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_a_call_reads_what_the_call_directly_before_it_wrote(m, dtype):
    """No torch operator between the calls: every result is the next call's input (f16: no conversion between them either) and residual, the
    gated result too, and a decode call reads the last; the same bits as with a wait behind every call."""
    cols = 1024  # weights of 0.01: a projection scales by 0.32, the gated product stays small, so 24 calls stay inside f16
    ws = [ctx().prepare_weight(t, H.random_weight(t, cols, cols, seed=260 + i, std=0.01), cols, cols) for i, t in enumerate((H.Q4_K, H.Q8_0, H.IQ4_NL, H.Q4_0))]
    x0 = torch.from_numpy(np.random.default_rng(261).standard_normal((m, cols)).astype(np.float32)).to("cuda", dtype)

    def chain(wait):
        x, outs = x0, []
        for i in range(8):
            x = ctx().linear(x, ws[i % 4], residual=x)
            if wait:
                ctx().sync()
            outs.append(x)
            g = ctx().gated_linear(x, ws[(i + 1) % 4], ws[(i + 1) % 4])
            if wait:
                ctx().sync()
            outs.append(g)
            x = ctx().linear(g, ws[(i + 2) % 4], residual=x)
            if wait:
                ctx().sync()
            outs.append(x)
            outs.append(ctx().linear(x[:4], ws[(i + 3) % 4]))
            if wait:
                ctx().sync()
        ctx().sync()
        return [o.float().cpu().numpy() for o in outs]

    want = chain(True)
    assert all(np.isfinite(o).all() for o in want)
    for _ in range(3):
        for a, b in zip(chain(False), want):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("m,epilogue_warps", [(24, 4), (64, 4), (96, 8), (128, 8), (200, 8)])
def test_gated_q6k_has_the_epilogue_warps_it_was_measured_with(gemm_variant, tmp_path, m, epilogue_warps):
    """Four up to 64 tokens per tile, where the dequantisers set the pace, eight above, where the epilogue does (2048 -> 8192 at 128 tokens 20.3 us with four, 17.8 with eight)."""
    from tests.test_gpu_row import launches_of

    if gemm_variant == "operand_pass":
        pytest.skip("the dequantising form")
    w = [ctx().prepare_weight(H.Q6_K, H.random_weight(H.Q6_K, 300, 512, seed=s), 300, 512) for s in (1, 2)]
    x = torch.randn((m, 512), device="cuda", dtype=torch.float16)
    (_, _, threads), = launches_of(lambda: ctx().gated_linear(x, *w), tmp_path, "gemm_kernel")
    assert threads == 32 * (3 + 16 + epilogue_warps)  # tokens, MMAs and packed boxes; the dequantisers


@pytest.mark.parametrize("tensor_type,cols,cut", [(H.Q8_0, 3328, False), (H.Q4_0, 2816, False), (H.Q6_K, 3328, True), (H.Q4_K, 11008, True)])
def test_short_tiles_are_cut_where_their_steps_take_longer_than_the_cut(gemm_variant, tmp_path, tensor_type, cols, cut):
    """30 tiles of 256 rows and 32 tokens: whole they are a pair each, cut they are everybody's.  Q8_0 3328 -> 7537 whole 11.0 us, cut 14.6."""
    from tests.test_gpu_row import launches_of

    if gemm_variant == "operand_pass":
        pytest.skip("the dequantising form")
    rows = 7537
    w = ctx().prepare_weight(tensor_type, H.random_weight(tensor_type, rows, cols, seed=1), rows, cols)
    x = torch.randn((32, cols), device="cuda", dtype=torch.float16)
    (_, ctas, _), = launches_of(lambda: ctx().linear(x, w), tmp_path, "gemm_kernel")
    assert ctas == (torch.cuda.get_device_properties(0).multi_processor_count // 2 * 2 if cut else 2 * 30)

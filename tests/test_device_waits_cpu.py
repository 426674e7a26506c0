"""Rules of the kernels' bounded waits that no run shows: a wait that gives up must not part a warp in front of an instruction that wants all of it.

What a kernel does after such a wait cannot be provoked without a fault, so the sources are read instead."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zllm_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _between(text, first, last):
    start = text.index(first)
    return text[start:text.index(last, start)]


def test_short_prefill_dequantisers_keep_the_warp_together():
    """tcgen05.st and tcgen05.wait::st are .sync.aligned: no lane may leave the loop between the waits and them."""
    roles = _source("zq_gemm.cu")
    body = _between(roles[roles.index("DqTensorRow{") - 1500:], "while (", "pair_arrive(")
    assert "wait_flag(" in body and "dq.emit(DqTensorRow{" in body
    assert not re.search(r"\b(break|return|continue)\b|while \(ok", body)
    assert body.count("ok = ok && wait_flag(") == body.count("wait_flag(") == 2


def test_short_prefill_issuers_leave_by_a_vote():
    """elect.sync and tcgen05.ld behind a wait: all lanes go on or none."""
    roles = _source("zq_gemm.cu")
    tokens = _between(roles, "const uint32_t sub = (uint32_t)p.box_tok * kBK * 2;", "elect_one()")
    assert "wait_warp<true>(&empty" in tokens
    mma = roles[roles.index("int before = 0;"):]
    mma = _between(mma, "if constexpr (SHORT)", "elect_one()")
    assert re.search(r"ok = __all_sync\(0xffffffffu, wait_flag\(&full.*wait_flag\(&a_full", mma)
    assert "wait_warp<SHORT>(&acc_empty" in roles and "wait_warp<SHORT>(&acc_full" in roles and "wait_warp<SHORT>(&p_empty" in roles


def test_streamed_row_groups_are_given_back_behind_their_sums():
    """The arrival that frees a ring stage must not overtake the loads from it: it stands behind the store of the sums that need them all."""
    kernel = _source("zq_gemv_row.cu")
    consumer = _between(kernel[kernel.index("gemv_row_stream_kernel(const"):], "row_unit<TYPE>(", "s += a.lanes_g;")
    assert consumer.count("mbar_arrive(&s_empty[s])") == 1
    assert consumer.index("at[8] = yacc[0][1];") < consumer.index("__syncwarp();") < consumer.index("mbar_arrive(&s_empty[s])")


def test_warps_leave_together_when_the_block_gives_up():
    """A lane may return by its own reading of the flag only where it is alone (`lane == 0` of the MoE copies)."""
    row, moe = _source("zq_gemv_row.cu"), _source("zq_moe_grouped.cu")
    assert "(volatile int *)&s_abort" not in row and row.count("if (i8_warp_aborts(&s_abort)) return;") == 3
    assert moe.count("(volatile int *)&s_abort") == 1 and len(re.findall(r"if \(i8_warp_aborts\(&s_abort\)\) return( false)?;", moe)) == 2
    copies = _between(moe, "if (warp == kI8Threads / 32) {", "if (warp > kI8Threads / 32)")
    assert copies.index("if (lane == 0) {") < copies.index("(volatile int *)&s_abort")

"""The native half of the host mirror where it needs no GPU: what it accepts and which exceptions come back.  A null context ends every
call in the C ABI's argument check."""
import numpy as np
import pytest
import torch


class StubWeight:
    _h, _rows, _cols = 1, 8, 4


def _native():
    from zllm_b200 import ffi

    return ffi.native()


@pytest.mark.parametrize("out_dtype", [None, torch.float32])
def test_batch_of_an_unreadable_dtype_is_a_key_error(out_dtype):
    with pytest.raises(KeyError) as info:
        _native().linear_batch(0, [(torch.zeros((2, 4), dtype=torch.float64), StubWeight())], out_dtype)
    assert info.value.args == (torch.float64,)


def test_host_batch_takes_an_output_marked_read_only():
    """The mark is numpy's and says nothing about the memory; it never was looked at."""
    from zllm_b200.ffi import ZqFailure

    y = np.zeros((2, 8), dtype=np.float32)
    y.flags.writeable = False
    with pytest.raises(ZqFailure, match="null"):  # arrived at the ABI
        _native().linear_host_batch(0, [(np.zeros((2, 4), dtype=np.float32), StubWeight(), y)])

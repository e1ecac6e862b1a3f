"""What the native host layer refuses, and with which exception: nothing of it reaches a kernel."""
import ctypes
import pathlib

import pytest
import torch

from dscuda_b200 import mla

pytestmark = pytest.mark.gpu


def _bf16(*shape):
    return torch.zeros(*shape, device="cuda", dtype=torch.bfloat16)


def _table():
    return torch.zeros(1, 1, device="cuda", dtype=torch.int32)


@pytest.mark.parametrize("call", [
    lambda: mla.mla_forward(_bf16(1, 1, 1, 2, 512), _bf16(1, 1, 2, 64), _bf16(1, 1, 512), _bf16(1, 1, 64), 0.1),
    lambda: mla.mla_decode(_bf16(1, 2, 576), _bf16(1, 64, 1, 576), _table(), _table()[0], 0.1),
    lambda: mla.cache_append(_bf16(1, 64, 1, 576), _bf16(1, 1, 1, 512), _bf16(1, 1, 64), _table()),
    lambda: mla.flash_forward(_bf16(1, 1, 1, 2, 128), _bf16(1, 1, 2, 128), _bf16(1, 1, 2, 128), 0.1),
    lambda: mla.prefill_forward(_bf16(4, 2, 128), _bf16(4, 2, 64), _bf16(4, 2, 128), _bf16(4, 1, 64), _bf16(4, 2, 128), 0.1),
    lambda: mla.absorb_query(_bf16(3, 0, 128), _bf16(0, 512)),
    lambda: mla.up_project(_bf16(3, 0), _bf16(256, 512), _bf16(256, 512), 2),
    lambda: mla.rope_apply(_bf16(1, 4, 0, 64)),
    lambda: mla.rope_apply(_bf16(4, 2, 64).transpose(0, 1), positions=_table()[0]),
], ids=["forward_5d", "decode_3d", "append_4d", "flash_5d", "dense_3d", "no_heads", "no_columns", "rope_no_heads", "strided"])
def test_refused_shapes(call):
    with pytest.raises(ValueError):
        call()


def test_tensor_without_storage():
    """data_ptr() throws between releasing the interpreter lock and taking it back."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        query, w = torch.empty(3, 2, 128, device="cuda", dtype=torch.bfloat16), torch.empty(256, 512, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        mla.absorb_query(query, w)


@pytest.mark.parametrize("longest", [37, 37.0, torch.tensor(37)])
def test_longest_sequence_as_any_number(longest):
    inputs = [torch.randn(37, heads, width, device="cuda").bfloat16() for heads, width in ((2, 128), (2, 64), (2, 128), (1, 64), (2, 128))]
    cu = torch.tensor([0, 37], device="cuda", dtype=torch.int32)
    packed = mla.prefill_forward(*inputs, 0.1, cu, longest)
    dense = mla.prefill_forward(*(x[None] for x in inputs), 0.1)
    assert torch.equal(packed[0], dense[0][0]) and torch.equal(packed[1], dense[1][0])


def test_a_refused_launch_leaves_no_error_behind():
    """The host refuses the launch (too many threads to a block); the next check of the caller's must not find its error."""
    lib = ctypes.CDLL(str(pathlib.Path(__file__).resolve().parents[1] / "build" / "libdscuda_test_probes.so"))
    assert lib.dscuda_test_failed_launch() == 0

"""What the native host layer checks about memory the caller brings, on tensors without storage: a call that passes the checks ends at the
first pointer, a call that does not is refused before it."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from dscuda_b200 import mla

BATCH, HEADS, SPLITS, SEQ = 2, 16, 8, 40
F32, BF16, I32, U8 = torch.float32, torch.bfloat16, torch.int32, torch.uint8


def fake(*shape, dtype=BF16, device="cuda:0"):
    with FakeTensorMode():
        return torch.empty(shape, dtype=dtype, device=device)


def strided(*shape, dtype=BF16):
    with FakeTensorMode():
        return torch.empty(*shape, 2, dtype=dtype, device="cuda:0")[..., 0]


def decode(splits=SPLITS, workspace=None, output=None, lse=None):
    return mla.mla_decode(fake(BATCH, 1, HEADS, 576), fake(4, 64, 1, 576), fake(BATCH, 2, dtype=I32), fake(BATCH, dtype=I32), 0.1, splits, workspace, output, lse)


def prefill(lead):
    return [fake(*lead, heads, width) for heads, width in ((HEADS, 128), (HEADS, 64), (HEADS, 128), (1, 64), (HEADS, 128))]


def forward(output=None, lse=None):
    return mla.prefill_forward(*prefill((BATCH, SEQ)), 0.1, output=output, lse=lse)


def backward(grads=None, workspace=None, packed=False):
    lead = (BATCH * SEQ,) if packed else (BATCH, SEQ)
    out = fake(*lead, HEADS, 128)
    layout = (fake(BATCH + 1, dtype=I32), SEQ) if packed else (None, None)
    return mla.prefill_backward(out, out, fake(BATCH * HEADS * SEQ, dtype=F32), *prefill(lead), 0.1, *layout, workspace=workspace, grads=grads)


def gradients(short=None):
    return [fake(BATCH * SEQ * heads * width - (1 if i == short else 0)) for i, (heads, width) in enumerate(((HEADS, 192), (HEADS, 128), (1, 64), (HEADS, 128)))]


def dequantise(first, rows, cache_rows=256, width=656):
    return mla.cache_dequantize_fp8(fake(4, 64, width, dtype=U8), fake(cache_rows, 576), first, rows)


ROWS = BATCH * HEADS
PARTIALS = ROWS * SPLITS * 514


@pytest.mark.parametrize("call", [
    lambda: decode(workspace=fake(PARTIALS - 1, dtype=F32)),
    lambda: decode(splits=SPLITS + 1, workspace=fake(PARTIALS, dtype=F32)),
    lambda: decode(workspace=fake(PARTIALS, dtype=F32, device="cuda:1")),
    lambda: decode(output=fake(ROWS * 512 - 1)),
    lambda: decode(output=fake(BATCH, 1, HEADS, 512, dtype=torch.float16)),
    lambda: decode(output=strided(BATCH, 1, HEADS, 512)),
    lambda: decode(output=fake(BATCH, 1, HEADS, 512, device="cuda:1")),
    lambda: decode(lse=fake(ROWS - 1, dtype=F32)),
    lambda: decode(lse=fake(ROWS, dtype=torch.float64)),
    lambda: forward(output=fake(BATCH * SEQ * HEADS * 128 - 1)),
    lambda: forward(lse=fake(BATCH * SEQ * HEADS - 1, dtype=F32)),
    lambda: backward(grads=gradients(short=0)),
    lambda: backward(grads=gradients(short=1)),
    lambda: backward(grads=gradients(short=2)),
    lambda: backward(grads=gradients(short=3), packed=True),
    lambda: backward(grads=[*gradients()[:3], strided(BATCH, SEQ, HEADS, 128)]),
    lambda: dequantise(0, 257, cache_rows=300),
    lambda: dequantise(200, 57, cache_rows=300),
    lambda: dequantise(1 << 40, 1, cache_rows=300),
    lambda: dequantise(0, 256, width=655),
    lambda: dequantise(200, 56, cache_rows=255),
], ids=["workspace", "more_splits", "workspace_device", "output", "output_dtype", "output_strided", "output_device", "lse", "lse_dtype", "forward_output",
        "forward_lse", "dq", "dk_nope", "dk_pe", "dv_packed", "dv_strided", "fp8_rows", "fp8_rows_behind_first", "fp8_first", "fp8_width", "cache_rows"])
def test_refused(call):
    with pytest.raises(ValueError):
        call()


def test_backward_workspace_of_a_lower_limit_is_refused():
    """The scratch limit belongs to the process: a workspace made under a lower one is too small once the limit is raised."""
    from dscuda_b200.library import library
    shape = (BATCH, SEQ, BATCH * SEQ, HEADS)
    previous = mla.prefill_backward_scratch_limit(0)
    try:
        low = library("mla").dscuda_mla_prefill_backward_workspace_bytes(*shape)
        mla.prefill_backward_scratch_limit(1 << 30)
        high = library("mla").dscuda_mla_prefill_backward_workspace_bytes(*shape)
        assert high > low
        for packed in (False, True):
            with pytest.raises(ValueError, match="workspace"):
                backward(grads=gradients(), workspace=fake(low, dtype=U8), packed=packed)
            with pytest.raises(ValueError, match="device"):
                backward(grads=gradients(), workspace=fake(high, dtype=U8, device="cuda:1"), packed=packed)
            with pytest.raises(RuntimeError, match="[Dd]river|data pointer|storage"):
                backward(grads=gradients(), workspace=fake(high, dtype=U8), packed=packed)
    finally:
        mla.prefill_backward_scratch_limit(previous)


def test_host_memory_is_refused():
    with pytest.raises(RuntimeError, match="no CPU path"):
        decode(output=torch.empty(BATCH, 1, HEADS, 512, dtype=BF16))


@pytest.mark.parametrize("call", [
    lambda: decode(),
    lambda: decode(workspace=fake(PARTIALS * 4, dtype=U8)),
    lambda: decode(workspace=fake(PARTIALS + 7, dtype=F32), output=fake(64, 1, HEADS, 512), lse=fake(64 * HEADS, dtype=F32)),
    lambda: forward(output=fake(BATCH * SEQ * HEADS * 128), lse=fake(BATCH * HEADS, SEQ, dtype=F32)),
    lambda: backward(grads=gradients()),
    lambda: backward(grads=gradients(), packed=True),
    lambda: dequantise(200, 56),
    lambda: dequantise(0, None),
], ids=["decode", "bytes", "larger", "forward", "dense", "packed", "rows", "all_rows"])
def test_what_fits_is_accepted(call):
    """The call gets past the checks: what ends it is the missing storage or, without a driver, the question for the stream."""
    with pytest.raises(RuntimeError, match="[Dd]river|data pointer|storage"):
        call()


@pytest.mark.parametrize("call", [
    lambda x: mla.up_project(x, fake(128, 512), fake(128, 512), 1),
    lambda x: mla.absorb_query(x, fake(128, 512)),
    lambda x: mla.unabsorb_output(x, fake(128, 512)),
    lambda x: mla.rope_apply(x),
], ids=["up_project", "absorb_query", "unabsorb_output", "rope"])
def test_tensor_without_dimensions(call):
    with pytest.raises(IndexError):
        call(fake())

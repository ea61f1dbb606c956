"""The allocation-free derivative needs no particular number of its blocks on the
GPU at once: it runs on a stream that owns a few SMs of the device (a green
context), with the values it gives on the whole device, and its launches are
ordinary ones that a graph replays there too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(r):
    assert int(r[0]) == 0, r[0]
    return r[1] if len(r) == 2 else r[1:]


@pytest.fixture(scope="module")
def few_sms():
    """A stream of 16 SMs."""
    import torch
    drv = pytest.importorskip("cuda.bindings.driver")

    torch.zeros(1, device="cuda")  # the primary context
    dev = _check(drv.cuDeviceGet(0))
    whole = _check(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    parts, n, _ = _check(drv.cuDevSmResourceSplitByCount(1, whole, 0, 16))
    assert n == 1 and parts[0].sm.smCount < whole.sm.smCount
    desc = _check(drv.cuDevResourceGenerateDesc([parts[0]], 1))
    ctx = _check(drv.cuGreenCtxCreate(desc, dev, drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    st = _check(drv.cuGreenCtxStreamCreate(ctx, drv.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield int(st)
    torch.cuda.synchronize()
    drv.cuStreamDestroy(st)
    drv.cuGreenCtxDestroy(ctx)


@pytest.mark.parametrize("shape", [(16, 16, 16), (96, 96, 96), (1024, 16, 16)])
def test_on_a_few_sms(qvti, few_sms, shape):
    import torch

    spacing = (10.0, 8.0, 12.0)
    f = np.random.default_rng(sum(shape)).standard_normal(shape).astype(np.float32)
    d_in = torch.from_numpy(f).cuda()
    want, out = torch.empty_like(d_in), torch.full_like(d_in, float("nan"))
    torch.cuda.synchronize()
    qvti.q_derivative_noalloc(d_in.data_ptr(), want.data_ptr(), shape, spacing, 1, True, 1, stream=0)
    torch.cuda.synchronize()
    qvti.q_derivative_noalloc(d_in.data_ptr(), out.data_ptr(), shape, spacing, 1, True, 1, stream=few_sms)
    torch.cuda.synchronize()
    assert torch.equal(out, want)

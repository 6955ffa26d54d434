"""solve_lp_device on a stream that owns a part of the GPU's SMs (a green context's): the cooperative launches of
the resident forms are sized for that part. The same bits as on a stream of the whole device, for LPs that fit the
part's shared memory, only the whole device's, and neither.
"""
import numpy as np
import pytest

import ps26119
from ps26119 import generators as g

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small_stream():
    import torch
    d = pytest.importorskip("cuda.bindings.driver")
    torch.zeros(1, device="cuda")  # the primary context

    def call(r):
        assert int(r[0]) == 0, r[0]
        return r[1] if len(r) == 2 else r[1:]

    dev = call(d.cuDeviceGet(0))
    sms = call(d.cuDeviceGetDevResource(dev, d.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    parts, _, _ = call(d.cuDevSmResourceSplitByCount(1, sms, 0, 32))
    assert parts[0].sm.smCount < sms.sm.smCount
    desc = call(d.cuDevResourceGenerateDesc([parts[0]], 1))
    ctx = call(d.cuGreenCtxCreate(desc, dev, d.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = call(d.cuGreenCtxStreamCreate(ctx, d.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield int(stream)
    d.cuStreamDestroy(stream)
    d.cuGreenCtxDestroy(ctx)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("rows", [5, 700, 10_000, 15_000, 60_000, 130_000])
def test_same_bits_as_on_the_whole_device(rows, precision, small_stream):
    import torch
    lp = g.random_lp(rows, min(rows, 7) if rows < 10 else None, min(rows, 6), seed=rows)
    names = ("c", "col_lower", "col_upper", "row_lower", "row_upper", "col_start", "row_index", "value")
    held = [torch.as_tensor(getattr(lp, k), device="cuda") for k in names]
    torch.cuda.synchronize()

    def solve(stream):
        out = [torch.empty(k, dtype=torch.float64, device="cuda") for k in (lp.num_cols, lp.num_rows, lp.num_cols)]
        torch.cuda.synchronize()
        r = ps26119.solve_lp_device(lp.num_rows, lp.num_cols, 1, 0.0, [t.data_ptr() for t in held],
                                    precision=precision, iteration_limit=192, stream=stream, out=[t.data_ptr() for t in out])
        torch.cuda.synchronize()
        return (r.status, r.iterations, r.message, r.objective), [t.cpu().numpy() for t in out]

    whole, part = solve(torch.cuda.Stream().cuda_stream), solve(small_stream)
    assert whole[0] == part[0]
    assert all(np.array_equal(a, b) for a, b in zip(whole[1], part[1]))

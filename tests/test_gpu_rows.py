"""Matrix-vector products of every format against exact sums, at the sizes where their row groups and passes end."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("fmt", ["f32", "f16", "bf16", "q4g32", "q4g64ref", "i8pc"])
@pytest.mark.parametrize("in_dim,out_dim,batch", [(64, 1, 1), (64, 7, 2), (576, 33, 1), (1088, 130, 8), (2112, 5, 11), (8192, 19, 4)])
def test_canonical_matvec(vb, oracle, fmt, in_dim, out_dim, batch):
    """Row remainders of the four-row groups, K of whole and ragged steps, passes of eight rows of x."""
    from velox_b200.engine import DeviceBuffer as dev
    c = {"f32": O.FMT_F32, "f16": O.FMT_F16, "bf16": O.FMT_BF16, "q4g32": O.FMT_Q4G32, "q4g64ref": O.FMT_Q4G64REF, "i8pc": O.FMT_I8PC}[fmt]
    w = oracle.fill_normal(out_dim * in_dim, 5, 1, 0.02).reshape(out_dim, in_dim)
    data, scales = oracle.quantize(w, c)
    x = oracle.fill_normal(batch * in_dim, 5, 2, 1.0).reshape(batch, in_dim)
    dw, dx, dy = dev.from_numpy(data), dev.from_numpy(x), dev(batch * out_dim * 4)
    ds = dev.from_numpy(scales) if scales is not None else None
    vb.check(vb.load().vb_op_matmul(dy.ptr, dx.ptr, dw.ptr, ds.ptr if ds else None, c, in_dim, out_dim, batch, None))
    got = dy.to_numpy(np.float32, (batch, out_dim))
    exact = x.astype(np.float64) @ oracle.dequantize(data, scales, c, out_dim, in_dim).astype(np.float64).T
    # fp32 sums of in_dim terms of std 0.02 each: in_dim roundings of 2^-24 of a partial sum below 5 * 0.02 * sqrt(in_dim)
    assert np.max(np.abs(got - exact)) <= in_dim * 2.0 ** -24 * 5 * 0.02 * np.sqrt(in_dim)

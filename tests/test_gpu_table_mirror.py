"""SPConvMM's table of a rulebook it is told is submanifold: read mirrored where the rulebook is symmetric, plainly where
it is not (another padding), with the same features as without the flag; narrow fp32 rows; the element-wise layer."""
import numpy as np
import pytest
import torch

from tests._util import assert_feats_close, rng
from tests.test_gpu_spconv import DEV, _t

pytestmark = pytest.mark.gpu
ONE, ZERO = (1, 1, 1), (0, 0, 0)


def _rulebook(d3d, n, shape, pad=ONE):
    ids = rng(n).choice(int(np.prod(shape)), n, replace=False)
    coors = np.stack(np.unravel_index(ids, shape), 1).astype(np.int32)
    num = torch.tensor([n], dtype=torch.int32, device=DEV)
    return num, d3d.spconv_index(_t(coors), num, torch.empty([1, 0] + shape[1:], dtype=torch.int32, device=DEV),
                                 (3, 3, 3), ONE, pad, ONE, ZERO, n, True, False)


@pytest.mark.parametrize("n,pad", [(160000, ONE), (160000, (1, 0, 1)), (400, ONE)])
def test_submanifold_flag_changes_nothing(d3d, n, pad):
    num, (index, num_index) = _rulebook(d3d, n, [1, 10, 240, 240], pad)
    x = torch.randn((n, 32), device=DEV).half()
    w = (rng(1).standard_normal((27, 32, 32)) * 0.05).astype(np.float32)
    got = d3d.spconv_mm(x, num, num, index, num_index, (3, 3, 3), 32, 32, n, True, False, w, None)
    want = d3d.spconv_mm(x, num, num, index, num_index, (3, 3, 3), 32, 32, n, False, False, w, None)
    assert torch.equal(got, want)


@pytest.mark.parametrize("cin,cout", [(1, 1), (4, 16), (16, 16), (17, 15), (16, 17), (33, 32), (64, 20)])
@pytest.mark.parametrize("n", [1, 129])
def test_narrow_fp32_rows(d3d, orc, cin, cout, n):
    num, (index, num_index) = _rulebook(d3d, n, [1, 5, 7, 8])
    x = rng(2).standard_normal((n, cin)).astype(np.float32)
    w = rng(3).standard_normal((27, cin, cout)).astype(np.float32)
    b = rng(4).standard_normal(cout).astype(np.float32)
    got = d3d.spconv_mm(_t(x), num, num, index, num_index, (3, 3, 3), cin, cout, n, True, False, w, b)
    want = orc.spconv_mm(x, w, b, index.cpu().numpy(), int(num_index.item()), False, n)
    assert_feats_close(got.cpu().numpy(), want, 1e-5)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [1, 7, 8, 4099])
@pytest.mark.parametrize("relu,with_res", [(1, False), (1, True), (2, True), (0, True)])
def test_activation(d3d, dtype, n, relu, with_res):
    from deploy3d_b200.plugins import activation
    x = torch.randn(n, device=DEV).to(dtype)
    r = torch.randn(n, device=DEV).to(dtype) if with_res else None
    want = torch.relu(x) if relu == 2 or not with_res else x
    want = want + r if with_res else want
    want = torch.relu(want) if relu == 1 else want
    assert torch.equal(activation(x.clone(), r, relu), want)

"""ReconBlock with concatenation and the gather back with labels, against the tensor operations they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TYPES = [torch.float16, torch.bfloat16, torch.float32]


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("rows,c", [(1, 8), (257, 64), (1000, 24)])
@pytest.mark.parametrize("copy_x", [False, True])
def test_recon(d3d, dtype, rows, c, copy_x):
    from deploy3d_b200.backbone import ew_apply
    from deploy3d_b200.plugins import recon
    a, b, g, x = (torch.randn((rows, c), device=DEV).mul_(3).to(dtype) for _ in range(4))
    out = torch.full((rows, 2 * c + 8), 7.0, device=DEV).to(dtype)
    recon(a, b, g, x, out, copy_x)
    want = ew_apply("recon", [t.float() for t in (a, b, g, x)], torch)
    tol = {torch.float32: 1e-6, torch.float16: 1e-3, torch.bfloat16: 8e-3}[dtype]
    torch.testing.assert_close(out[:, :c].float(), want, rtol=tol, atol=1e-6)
    assert torch.equal(out[:, c:2 * c], x if copy_x else torch.full_like(x, 7.0)) and (out[:, 2 * c:] == 7).all()


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("classes,ld", [(1, 8), (20, 32), (17, 17), (128, 128)])
@pytest.mark.parametrize("n", [1, 64, 65, 1000])
def test_gather_labels(d3d, dtype, classes, ld, n):
    from deploy3d_b200.plugins import gather_labels
    m = 300
    feats = torch.randn((m, ld), device=DEV).mul_(4).round_().to(dtype)[:, :classes]  # equal maxima on purpose
    ids = torch.randint(-2, m + 2, (n,), dtype=torch.int32, device=DEV)
    logits = torch.empty((n, classes), device=DEV)
    labels = torch.empty(n, dtype=torch.int32, device=DEV)
    gather_labels(feats, ids, 0.25, logits, labels)
    ok = (ids >= 0) & (ids < m)
    want = torch.where(ok[:, None], feats[ids.clamp(0, m - 1).long()].float(), torch.tensor(0.25, device=DEV))
    assert torch.equal(logits, want)
    first = (want == want.max(1, keepdim=True).values).int().argmax(1)
    assert torch.equal(labels.long(), first.long())

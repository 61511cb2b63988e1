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


def _small_net(layers, order, feats):
    """Runs a network of submanifold layers over 300 voxels; its features."""
    from deploy3d_b200.backbone import SparseNet
    ids = torch.arange(300, device=DEV) * 7
    coors = torch.stack([0 * ids, ids // 400, ids // 20 % 20, ids % 20], 1).int()
    net = SparseNet(layers, [1, 8, 20, 20], {"in": 300}, dtype=torch.float16, device=DEV, plugin_order=order)
    net.set_input(coors, torch.tensor([300], dtype=torch.int32, device=DEV))
    return net.forward(feats)[0].clone()


def _features(layout):
    x = torch.randn((300, 16), generator=torch.Generator(device=DEV).manual_seed(3), device=DEV).half()
    if layout == "columns":  # of a wider tensor
        wide = torch.full((300, 24), 9.0, device=DEV).half()
        wide[:, :16] = x
        return wide[:, :16]
    if layout == "offset":  # rows that start two bytes behind a multiple of 16
        flat = torch.full((300 * 16 + 1,), 9.0, device=DEV).half()
        flat[1:] = x.reshape(-1)
        return flat[1:].view(300, 16)
    return x


@pytest.mark.parametrize("act_first", [False, True])
def test_residual_with_strides_of_its_own(d3d, act_first):
    """The caller's features as a residual in plugin order, columns of a wider tensor."""
    from deploy3d_b200.backbone import Layer
    layers = [Layer("subm", "a", 16, 16, residual="input", act_first=act_first)]
    want = _small_net(layers, True, _features("rows"))
    assert torch.equal(_small_net(layers, True, _features("columns")), want)


def test_recon_of_features_with_strides_of_their_own(d3d):
    from deploy3d_b200.backbone import Layer
    layers = [Layer("subm", "a", 16, 16, save="a", source="input", relu=False),
              Layer("ew", None, 16, 16, ew=("recon", ["a", "a", "a", "input"]), save="r"),
              Layer("ew", None, 16, 32, ew=("concat", ["r", "input"]), save="c")]
    want, got = (_small_net(layers, True, _features(f)).float() for f in ("rows", "columns"))
    # one fp16 rounding of values that differ by the fp32 rounding of the sigmoids: half an ulp either way
    assert (got - want).abs().max() <= 2 ** -10 * want.abs().max() and torch.equal(got[:, 16:], want[:, 16:])


def test_element_wise_passes_refuse_what_they_cannot_read(d3d):
    from deploy3d_b200.plugins import activation, recon
    x, y = _features("rows"), _features("columns")
    with pytest.raises(ValueError):
        activation(x.clone(), y)
    with pytest.raises(ValueError):
        activation(y)
    with pytest.raises(ValueError):
        recon(x, x, x, _features("offset"), out=x.clone())

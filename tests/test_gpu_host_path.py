"""The native enqueue and the operator layer's plugin look-up: what is kept between calls never outlives its inputs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("cin,cout,dtype", [(16, 16, torch.float32), (32, 64, torch.float16)])
def test_changed_weights_are_seen(d3d, cin, cout, dtype):
    """The same array objects with new contents, and other arrays with the same contents, give what fresh ones give."""
    r = np.random.Generator(np.random.PCG64(3))
    n = 700
    grid = (8, 20, 20)
    ids = r.choice(8 * 20 * 20, n, replace=False)
    coors = np.stack([0 * ids, ids // 400, ids // 20 % 20, ids % 20], 1).astype(np.int32)
    num = torch.tensor([n], dtype=torch.int32, device=DEV)
    one = (1, 1, 1)
    index, num_index = d3d.spconv_index(torch.from_numpy(coors).to(DEV), num,
                                        torch.empty((1, 0) + grid, dtype=torch.int32, device=DEV), (3, 3, 3), one, one,
                                        one, (0, 0, 0), n, True, False)
    x = torch.randn((n, cin), device=DEV).to(dtype)

    def run(w, b):
        return d3d.spconv_mm(x, num, num, index, num_index, (3, 3, 3), cin, cout, n, True, False, w, b).clone()

    w = r.standard_normal((27, cin, cout)).astype(np.float32)
    b = r.standard_normal(cout).astype(np.float32)
    first = run(w, b)
    assert torch.equal(first, run(w, b)) and torch.equal(first, run(w.copy(), b.copy()))
    old = w[26, cin - 1, cout - 1]
    w[26] *= -1  # the last offset only: the compare has to reach the end
    changed = run(w, b)
    assert torch.equal(changed, run(w.copy(), b)) and not torch.equal(changed, first)
    w[26] *= -1
    assert w[26, cin - 1, cout - 1] == old and torch.equal(first, run(w, b))
    b[cout - 1] += 1
    moved = run(w, b)
    assert torch.equal(moved[:, :-1], first[:, :-1]) and not torch.equal(moved[:, -1], first[:, -1])
    assert torch.equal(moved, run(np.asfortranarray(w), b.copy()))  # a layout that is not the blob's


def test_shapes_and_types_in_turn(d3d):
    """More signatures than a plugin keeps, the first of them again at the end."""
    pts = [torch.randn((5 + i, 3 + i % 4), device=DEV) for i in range(12)]
    to = [torch.arange(len(p), dtype=torch.int32, device=DEV).flip(0) for p in pts]
    for _ in range(2):
        for p, t in zip(pts, to):
            assert torch.equal(d3d.gather_back(p, t, 0.0), p.flip(0))
            h = p.half()
            assert d3d.gather_back(h, t, 0.0).dtype == torch.float16
    neg = torch.full((4,), -1, dtype=torch.int32, device=DEV)
    assert torch.signbit(d3d.gather_back(pts[0], neg, -0.0)).all()
    assert not torch.signbit(d3d.gather_back(pts[0], neg, 0.0)).any()


def test_refusals(d3d):
    from deploy3d_b200._lib import D3DError
    with pytest.raises(RuntimeError, match="CUDA tensors"):
        d3d.gather_back(torch.zeros((3, 2)), torch.zeros(3, dtype=torch.int32))
    with pytest.raises(TypeError, match="dtype"):
        d3d.gather_back(torch.zeros((3, 2), dtype=torch.float64, device=DEV),
                        torch.zeros(3, dtype=torch.int32, device=DEV))
    with pytest.raises(D3DError):
        d3d.nms3d(torch.zeros((1, 4), device=DEV), torch.zeros((1, 4, 5), device=DEV))


def test_nms_calls_share_no_mask(d3d):
    """nms3d runs with a mask of its own: not with one that a call in another thread has just installed in the plugin
    both use, whatever moment the threads switch at."""
    from deploy3d_b200 import synth
    from deploy3d_b200.ops import decoder
    case = synth.config4_boxes(2, 300)
    scores, boxes = (torch.from_numpy(case[k]).to(DEV) for k in ("scores", "boxes"))
    want = d3d.nms3d(scores, boxes, 0.17)
    plug = decoder._NMS[0.17]
    others = torch.full((1 << 20,), 77, dtype=torch.uint8, device=DEV)
    plug.__class__ = type("Contended", (type(plug),), {"_workspace": property(lambda s: others, lambda s, v: None)})
    try:
        assert torch.equal(d3d.nms3d(scores, boxes, 0.17), want)
        assert (others == 77).all()
    finally:
        del decoder._NMS[0.17]


def test_other_shapes_between_the_steps_of_a_call(d3d):
    """The caller's `outputs` may be any iterable; one that calls the same plugin with more shapes than it keeps does not
    change what its own call runs with."""
    from deploy3d_b200.plugins import deserialize_plugin
    plug = deserialize_plugin("NMS3d", b"")
    case = [torch.rand((1, 400), device=DEV).sort(descending=True)[0], torch.rand((1, 400, 7), device=DEV) + 1]
    want = plug.enqueue(*case)[0]

    class Outputs:
        def __iter__(self):
            for k in range(1, 10):  # nine smaller shapes, the workspace with them
                plug.enqueue(case[0][:, :k], case[1][:, :k])
            plug._workspace = None
            return iter([out])

    for _ in range(9):
        out = torch.zeros_like(want)
        assert plug.enqueue(*case, outputs=Outputs())[0] is out and torch.equal(out, want)


def test_missing_and_unreachable_tensors_are_refused(d3d):
    """What would become a null or a host address in a kernel is an error; an output without elements, a shape on the host
    and pinned memory are not."""
    from deploy3d_b200.plugins import deserialize_plugin
    nms = deserialize_plugin("NMS3d", b"")
    scores, boxes = torch.rand((1, 70), device=DEV).sort(descending=True)[0], torch.rand((1, 70, 7), device=DEV) + 1
    want, = nms.enqueue(scores, boxes)
    with pytest.raises(ValueError, match="0 of 1 outputs"):
        nms.enqueue(scores, boxes, outputs=[])
    with pytest.raises(RuntimeError, match="input 1 is not in CUDA memory"):
        nms.enqueue(scores, boxes.cpu())
    with pytest.raises(RuntimeError, match="output 0 is not in CUDA memory"):
        nms.enqueue(scores, boxes, outputs=[torch.zeros_like(scores, device="cpu")])
    assert torch.equal(nms.enqueue(scores, boxes.cpu().pin_memory())[0], want)

    blob = d3d.data_s_spconv_index((3, 3, 3), (2, 2, 2), (1, 1, 1), (1, 1, 1), (0, 0, 0), 50, False, False)
    plug = deserialize_plugin("SPConvIdx3d", blob)
    ids = torch.arange(60)
    coors = torch.stack([0 * ids, ids // 20, ids % 20, ids % 7], 1).int().to(DEV)
    num = torch.tensor([60], dtype=torch.int32, device=DEV)
    want = plug.enqueue(coors, num, torch.empty((1, 0, 4, 20, 8), dtype=torch.int32, device=DEV))
    outs = [torch.empty_like(t) for t in want[:4]]  # without the shape carrier, which has no elements
    got = plug.enqueue(coors, num, torch.empty((1, 0, 4, 20, 8), dtype=torch.int32), outputs=outs)
    assert len(got) == 4 and torch.equal(got[0], want[0]) and torch.equal(got[3], want[3])
    with pytest.raises(ValueError, match="3 of 5 outputs"):
        plug.enqueue(coors, num, torch.empty((1, 0, 4, 20, 8), dtype=torch.int32), outputs=outs[:3])

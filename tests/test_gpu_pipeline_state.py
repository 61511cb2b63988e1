"""What the frame pipelines and networks keep between their calls, on a small detection frame."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _frame(n=4000, seed=7):
    from deploy3d_b200 import synth
    frame = synth.config3_points()
    r = np.random.Generator(np.random.PCG64(seed))
    pts = frame["points"][r.permutation(len(frame["points"]))[:n]]
    return dict(points=np.ascontiguousarray(pts), batch=np.zeros(n, np.int32))


def _pipe(frame, device=DEV, caps=None, **how):
    from deploy3d_b200.pipeline import DetectionPipeline
    n = len(frame["points"])
    caps = caps or {"in": n, "down2": 8 * n, "down3": 8 * n, "down4": 8 * n, "out": 8 * n}
    pipe = DetectionPipeline("second", device, n_class=1, topk=64, n_pts=n, caps=caps, **how)
    pipe.load_frame(frame)
    return pipe


def _run(pipe):
    feats, coors, num = pipe.enqueue()
    torch.cuda.synchronize()
    n = int(num.item())
    return feats[:n].float(), coors[:n].clone(), pipe.net.counts(), pipe.bev.float()


def _assert_same_frame(got, want):
    """Features to the order of the encoder's atomic sums (fp32, rounded to fp16 in 12 layers)."""
    assert got[2] == want[2]
    assert torch.equal(got[1], want[1])
    for a, b in ((got[0], want[0]), (got[3], want[3])):
        assert (a - b).norm() <= 1e-2 * b.norm()


def test_device_without_an_index(d3d):
    frame = _frame()
    want = _run(_pipe(frame))
    assert min(want[2].values()) > 100
    pipe = _pipe(frame, device="cuda")
    for _ in range(2):
        _assert_same_frame(_run(pipe), want)


@pytest.mark.parametrize("small", [None, "in", "down2", "down4"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_lost_voxels_are_reported(d3d, small, dtype):
    """A frame whose voxels do not fit one of the buffers sets the pipeline's status word, eagerly and from the graph."""
    frame = _frame()
    caps = {k: v + 5 for k, v in _run(_pipe(frame))[2].items()}
    if small:
        caps[small] -= 6
    pipe = _pipe(frame, caps=caps, dtype=dtype)
    _run(pipe)
    assert int(pipe.status.item()) == (2 if small else 0)  # D3D_STATUS_OUTPUT_OVERFLOW
    pipe.capture()
    pipe.status.zero_()
    pipe.replay()
    torch.cuda.synchronize()
    assert int(pipe.status.item()) == (2 if small else 0)


def test_reading_a_rulebook_leaves_the_cleared_tables_alone(d3d):
    """The rulebook of a strided layer is made on demand; between `begin` and `forward` that must not touch the look-up that
    `begin` has cleared for the tables."""
    frame = _frame()
    want = _run(_pipe(frame))
    pipe = _pipe(frame)
    _run(pipe)
    net = pipe.net
    net.begin()
    read = {k: net.rulebooks[k].index.clone() for k in ("down2", "down3", "out")}
    feats, coors, num = net.forward(pipe.vox_feats_lp)
    torch.cuda.synchronize()
    assert net.counts() == want[2] and torch.equal(coors[:int(num)], want[1])
    for k, index in read.items():
        assert torch.equal(net.rulebooks[k].index, index)


@pytest.mark.parametrize("room", [1.2, 1.0, 0.6])
def test_rulebook_of_the_live_voxel_set(d3d, orc, room):
    """The rulebook of a strided layer lists the pairs between the voxels the network has, also where a set has lost some."""
    frame = _frame()
    caps = {k: (v + 9 if k == "in" else max(1, int(v * room))) for k, v in _run(_pipe(frame))[2].items()}
    pipe = _pipe(frame, caps=caps)
    _run(pipe)
    for key in ("down2", "down4", "out"):
        rb = pipe.net.rulebooks[key]
        src, dst = ({k: v.cpu().numpy() for k, v in pipe.net.sets[s].items() if k in ("coors", "num")}
                    for s in (rb.in_set, rb.out_set))
        index, num = rb.index.cpu().numpy(), int(rb.num_index.item())
        orc.check_layout(index, num, rb.kvol)
        inputs, outputs = src["coors"][:src["num"][0]], dst["coors"][:dst["num"][0]]
        ids = {tuple(c): i for i, c in enumerate(outputs.tolist())}
        taps = np.stack(np.meshgrid(*[np.arange(k) for k in rb.ksize], indexing="ij"), -1).reshape(-1, 3)
        want = set()
        for i, c in enumerate(inputs):
            at = c[1:] + np.array(rb.padding) - taps
            for k in np.flatnonzero(((at % np.array(rb.stride)) == 0).all(1)):
                o = ids.get((int(c[0]),) + tuple((at[k] // np.array(rb.stride)).tolist()))
                if o is not None:
                    want.add((i, o, int(k)))
        live = index[:, :num][:, index[2, :num] >= 0]
        assert len(want) == live.shape[1] > 100 and set(map(tuple, live.T.tolist())) == want


def test_clear_outside_a_graph_is_no_part_of_it(d3d):
    """`begin` before a capture and `forward` inside it: the graph clears for itself, on every replay; and a clear that a
    graph has recorded is not taken for one that has run."""
    frame = _frame()
    want = _run(_pipe(frame))
    pipe = _pipe(frame)
    _run(pipe)
    net, graph = pipe.net, torch.cuda.CUDAGraph()
    net.begin()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        feats, coors, num = net.forward(pipe.vox_feats_lp)
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        assert net.counts() == want[2] and torch.equal(coors[:int(num)], want[1])
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        net.begin()
        torch.cuda.current_stream().wait_stream(net.side)
        torch.cuda.current_stream().wait_stream(net.side_subm)
    _, coors, num = net.forward(pipe.vox_feats_lp)
    torch.cuda.synchronize()
    assert net.counts() == want[2] and torch.equal(coors[:int(num)], want[1])

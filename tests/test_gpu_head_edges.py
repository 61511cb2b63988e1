"""NMS3d and YoloX3dDecode where their kernels split: 64-box blocks, the finer grid of small calls, the sweep's limit of
2048 boxes, long chains of suppressions, boxes the cheap rejections must leave alone; maps a cluster cannot hold, as
many candidates as the kernel takes, equal scores everywhere."""
import numpy as np
import pytest
import torch

from tests._util import rng
from tests.test_gpu_decoder import _check, _head

pytestmark = pytest.mark.gpu


def _nms(d3d, orc, boxes, thr):
    b, k = boxes.shape[:2]
    scores = np.tile(1 - np.arange(k, dtype=np.float32) / (k + 1), (b, 1))
    got = d3d.nms3d(torch.from_numpy(scores).cuda(), torch.from_numpy(boxes).cuda(), thr).cpu().numpy()
    assert (got == orc.nms3d(scores, boxes, thr)).all()
    return got


def _boxes(r, b, k, spread):
    return np.concatenate([r.standard_normal((b, k, 3)) * spread, r.uniform(0.5, 5, (b, k, 3)),
                           r.uniform(-np.pi, np.pi, (b, k, 1))], -1).astype(np.float32)


@pytest.mark.parametrize("b,k", [(1, 63), (5, 64), (1, 129), (2, 960), (9, 961), (1, 2048), (1, 2049)])
@pytest.mark.parametrize("thr", [0.05, 0.7])
def test_nms_block_edges(d3d, orc, b, k, thr):
    _nms(d3d, orc, _boxes(rng(k), b, k, 4.0 + k / 50), thr)


def test_nms_chain_of_suppressions(d3d, orc):
    """Every box suppresses exactly the next one: no two of a block are decided in the same round."""
    boxes = np.zeros((1, 300, 7), np.float32)
    boxes[0, :, 0] = np.arange(300) * 1.0
    boxes[0, :, 3:6] = 2.0
    got = _nms(d3d, orc, boxes, 0.2)
    assert ((got[0] >= 0) == (np.arange(300) % 2 == 0)).all()


@pytest.mark.parametrize("case", ["identical", "axis_aligned_grid", "millimetres", "far_out", "negative_extent", "touching"])
def test_nms_boxes_the_rejections_must_not_touch(d3d, orc, case):
    r = rng(7)
    boxes = _boxes(r, 2, 200, 3.0)
    if case == "identical":  # up to 24 hull points per pair
        boxes[:] = boxes[:, :1]
        boxes[:, 100:, 6] += np.float32(np.pi / 2)
    elif case == "axis_aligned_grid":  # shared corners and collinear edges
        boxes[..., :2] = np.round(boxes[..., :2])
        boxes[..., 3:5] = np.ceil(boxes[..., 3:5])
        boxes[..., 6] = 0
    elif case == "millimetres":
        boxes[..., :6] *= np.float32(1e-3)
    elif case == "far_out":
        boxes[..., :2] += np.float32(5e4)
    elif case == "negative_extent":
        boxes[:, 1::3, 4] *= -1
    else:  # overlaps of a few hundredths, around the threshold
        boxes[..., 6] = np.float32(0.3)
        boxes[..., 3:5] = 2
        boxes[..., :2] *= np.float32(4)
    for thr in (0.01, 0.1, 0.5):
        _nms(d3d, orc, boxes, thr)


@pytest.mark.parametrize("dtype", ["fp32", "fp16"])
@pytest.mark.parametrize("size,topk,ties", [(512, 300, False), (443, 4096, False), (100, 4096, True), (7, 1, True)])
def test_decode_map_and_topk_edges(d3d, orc, size, topk, ties, dtype):
    scores, preds = _head(rng(size + topk), 1, 2, size, size + 1, 0, ties)
    _check(d3d, orc, scores, preds, np.array([0, -40, -3, 0.1, 0.1, 4], np.float32), 4, (1, 2), topk, dtype)


def test_decode_all_scores_equal(d3d, orc):
    scores, preds = _head(rng(3), 2, 1, 90, 70, 0)
    scores[:] = 0.25
    _check(d3d, orc, scores, preds, np.array([0, -40, -3, 0.1, 0.1, 4], np.float32), 4, (0,), 777, "fp32")

"""The rulebook kernels for 3-D kernels of at most three taps per axis: every lookup they choose between (the grid itself,
bit map + hash table, hash table), block edges, truncation, and the neighbour tables built without the rulebook."""
import numpy as np
import pytest
import torch

from tests._util import assert_table_consistent, assert_tables_equal, rng, table_pairs, table_parts, unique_coors
from tests.test_gpu_spconv import DEV, _t, check_index, run_index

pytestmark = pytest.mark.gpu
ONE, ZERO = (1, 1, 1), (0, 0, 0)
GRIDS = {"direct": [1, 9, 20, 21], "bits": [2, 40, 160, 150], "hash": [1, 41, 1600, 1408]}


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 600])
@pytest.mark.parametrize("ks,dil", [((3, 3, 3), ONE), ((1, 3, 3), (1, 2, 1)), ((3, 1, 2), (3, 1, 2)), ((2, 3, 1), ONE)])
def test_subm_rulebook(d3d, orc, grid, n, ks, dil):
    shape = GRIDS[grid]
    coors = unique_coors(rng(n), n, shape) if np.prod(shape) < 1 << 24 else \
        np.unique(np.stack([rng(n + d).integers(0, s, n) for d, s in enumerate(shape)], 1), axis=0).astype(np.int32)
    coors[: n // 2, 1:] = coors[: n // 2, 1:] // 4  # some of them crowded, so that neighbours exist
    coors = np.unique(coors, axis=0)
    coors = coors[rng(1).permutation(len(coors))]
    pd = tuple(d * (k // 2) for k, d in zip(ks, dil))
    n_max = len(coors) + (0 if n % 2 else 77)
    outs, _ = run_index(d3d, coors, n_max, [shape[0], 0] + shape[1:], ks, ONE, pd, dil, ZERO, n_max, True, False)
    check_index(orc, outs, coors, n_max, shape, ks, ONE, pd, dil, ZERO, n_max, True, False)


@pytest.mark.parametrize("grid", ["direct", "bits"])
def test_subm_rulebook_with_duplicates_and_stray_voxels(d3d, orc, grid):
    """Voxels that occur twice (the smaller index stands for both) and coordinates outside the grid."""
    shape = GRIDS[grid]
    coors = unique_coors(rng(5), 400, shape)
    coors[200:300] = coors[:100]
    coors[350:360, 3] = shape[3] + 5
    coors[360:365, 0] = -1
    outs, _ = run_index(d3d, coors, 400, [shape[0], 0] + shape[1:], (3, 3, 3), ONE, ONE, ONE, ZERO, 400, True, False)
    first = {}
    for i, c in enumerate(map(tuple, coors.tolist())):
        if all(0 <= v < e for v, e in zip(c, shape)):
            first.setdefault(c, i)
    index, num = outs[0].cpu().numpy(), int(outs[1].item())
    orc.check_layout(index, num, 27)
    for k in range(27):
        tap = np.array([0, k // 9, k // 3 % 3, k % 3]) - [0, 1, 1, 1]
        pairs = [(i, first[c]) for i, c in enumerate(map(tuple, (coors - tap).tolist())) if c in first]
        got = index[:2, :num][:, index[2, :num] == k].T
        assert got.tolist() == [list(p) for p in pairs], k


CONVS = [((3, 3, 3), (2, 2, 2), ONE, ONE, False), ((3, 1, 1), (2, 1, 1), ZERO, ONE, False),
         ((3, 3, 3), ONE, ONE, ONE, False), ((3, 3, 3), (2, 2, 1), ONE, (2, 1, 1), False),
         ((2, 2, 2), (2, 2, 2), ZERO, ONE, True), ((3, 3, 3), (3, 2, 1), ONE, ONE, True)]


@pytest.mark.parametrize("n", [1, 256, 257, 1500])
@pytest.mark.parametrize("ks,st,pd,dil,tr", CONVS)
@pytest.mark.parametrize("room", [1.0, 0.3])
def test_conv_rulebook(d3d, orc, n, ks, st, pd, dil, tr, room):
    shape = [2, 13, 24, 25]
    coors = unique_coors(rng(n), n, shape)
    m = orc.rulebook_conv(coors, shape, ks, st, pd, dil, ZERO, tr, 10 ** 7, max_num_act_in=n)[3]
    max_out = max(1, int(m * room))
    outs, _ = run_index(d3d, coors, n, [2, 0] + shape[1:], ks, st, pd, dil, ZERO, max_out, False, tr)
    check_index(orc, outs, coors, n, shape, ks, st, pd, dil, ZERO, max_out, False, tr)
    assert int(outs[3].item()) == min(m, max_out)


def test_conv_numbering_is_by_first_touch_across_many_blocks(d3d):
    """A thousand blocks: the numbers are those of a serial walk over the inputs and, for each, over the offsets."""
    shape, n = [1, 21, 400, 352], 300000
    coors = unique_coors(rng(8), n, shape)
    outs, _ = run_index(d3d, coors, n, [1, 0] + shape[1:], (3, 3, 3), (2, 2, 2), ONE, ONE, ZERO, 600000, False, False)
    tap = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(27, 3)
    at = coors[:, None, 1:] + 1 - tap[None]
    ok = ((at % 2 == 0) & (at >= 0) & (at // 2 < np.array([11, 200, 176]))).all(-1)
    key = ((at[..., 0] // 2 * 200 + at[..., 1] // 2) * 176 + at[..., 2] // 2)[ok]
    _, first = np.unique(key, return_index=True)
    want = key[np.sort(first)]
    m = int(outs[3].item())
    got = outs[2].cpu().numpy()[:m]
    assert m == len(want) and ((got[:, 1] * 200 + got[:, 2]) * 176 + got[:, 3] == want).all()


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("n", [1, 128, 129, 400])
def test_subm_tables_of_several_kernels(d3d, grid, n):
    from deploy3d_b200.plugins import SPConvMMPlugin, SubmTables
    shape, cap = GRIDS[grid], 500
    coors = np.zeros((cap, 4), np.int32)
    coors[:n] = unique_coors(rng(n), n, [shape[0], 9, 12, 13])
    coors_t, num = _t(coors), torch.tensor([n], dtype=torch.int32, device=DEV)
    shp = torch.empty([shape[0], 0] + shape[1:], dtype=torch.int32, device=DEV)
    kernels = [(3, 3, 3), (1, 3, 3), (3, 1, 3), (3, 1, 1), (1, 3, 1), (1, 1, 3), (1, 1, 1)]
    for sub in (kernels, kernels[1:2], kernels[3:5]):
        vols = [int(np.prod(k)) for k in sub]
        tables = [torch.full((SPConvMMPlugin.table_bytes(v, cap),), 93, dtype=torch.uint8, device=DEV) for v in vols]
        SubmTables(sub).enqueue(coors_t, num, shp, tables=tables)
        for k, v, t in zip(sub, vols, tables):
            index, num_index = d3d.spconv_index(coors_t, num, shp, k, ONE, tuple(x // 2 for x in k), ONE, ZERO, cap,
                                                True, False)
            want = SPConvMMPlugin.prepare(v, False, cap, index, num_index)
            got = table_parts(t, v, cap)
            assert_tables_equal(got, table_parts(want, v, cap), "%s" % (k,))
            assert_table_consistent(*got)


def _conv_tables_expected(d3d, coors, num, shp, out_shape, params, max_out):
    """Output voxels in cell order and the (output, offset, input) triples of a strided kernel, from its rulebook: of more
    than max_out outputs the first are kept."""
    index, num_index, oc, on, _ = d3d.spconv_index(coors, num, shp, *params[:4], ZERO, 200000, False, params[4])
    m, o = int(on.item()), [int(v) for v in out_shape]
    oc = oc[:m].long()
    key = ((oc[:, 0] * o[1] + oc[:, 1]) * o[2] + oc[:, 2]) * o[3] + oc[:, 3]
    order = torch.argsort(key)
    ids = torch.empty_like(order)
    ids[order] = torch.arange(m, device=DEV)
    pairs = index[:, :int(num_index.item())].long()
    pairs = pairs[:, pairs[2] >= 0]
    trip = torch.stack([ids[pairs[1]], pairs[2], pairs[0]], 1)
    return m, oc[order][:max_out].int(), trip[trip[:, 0] < max_out]


def _sorted(trip):
    return trip[torch.argsort((trip[:, 0] * 64 + trip[:, 1]) * (1 << 32) + trip[:, 2])]


def _conv_tables(d3d, plug, coors, num, shp, max_out, kvol, **how):
    from deploy3d_b200.plugins import SPConvMMPlugin
    cap = coors.shape[0]
    fwd = torch.full((SPConvMMPlugin.table_bytes(kvol, max_out),), 55, dtype=torch.uint8, device=DEV)
    inv = torch.full((SPConvMMPlugin.table_bytes(kvol, cap),), 55, dtype=torch.uint8, device=DEV)
    oc, on = torch.zeros((max_out, 4), dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    if how.get("cleared"):
        plug.tables_clear(coors, num, shp, table=None if how.get("voxel_grid") else fwd, device=DEV)
    plug.tables(coors, num, shp, out_coors=oc, num_act_out=on, table=fwd, table_inverse=inv, **how)
    return oc, on, table_parts(fwd, kvol, max_out), table_parts(inv, kvol, cap)


def _check_conv_tables(got, want, max_out):
    (oc, on, fwd, inv), (m, want_oc, trip) = got, want
    live = min(m, max_out)
    assert int(on.item()) == live and torch.equal(oc[:live], want_oc)
    assert_table_consistent(*fwd)
    assert_table_consistent(*inv)
    assert torch.equal(table_pairs(fwd), _sorted(trip))
    assert torch.equal(table_pairs(inv), _sorted(trip[:, [2, 1, 0]]))


def _out_shape(shape, ks, st, pd, dil, tr):
    if tr:
        return [shape[0]] + [(e - 1) * s - 2 * p + (k - 1) * d + 1 for e, k, s, p, d in zip(shape[1:], ks, st, pd, dil)]
    return [shape[0]] + [(e + 2 * p - d * (k - 1) - 1) // s + 1 for e, k, s, p, d in zip(shape[1:], ks, st, pd, dil)]


def _carrier(shape):
    return torch.empty([shape[0], 0] + list(shape[1:]), dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("ks,st,pd,dil,tr", CONVS)
@pytest.mark.parametrize("n,room", [(1, 1.0), (700, 1.3), (700, 0.4)])
def test_conv_tables(d3d, ks, st, pd, dil, tr, n, room):
    from deploy3d_b200.plugins import deserialize_plugin
    shape, cap, kvol = [1, 13, 24, 25], 750, int(np.prod(ks))
    coors = np.zeros((cap, 4), np.int32)
    coors[:n] = unique_coors(rng(n), n, shape)
    coors_t, num, shp = _t(coors), torch.tensor([n], dtype=torch.int32, device=DEV), _carrier(shape)
    params, out = (ks, st, pd, dil, tr), _out_shape(shape, ks, st, pd, dil, tr)
    max_out = max(1, int(_conv_tables_expected(d3d, coors_t, num, shp, out, params, 1)[0] * room))
    plug = deserialize_plugin("SPConvIdx3d", d3d.data_s_spconv_index(ks, st, pd, dil, ZERO, max_out, False, tr))
    assert plug.tables_ok(coors_t, num, shp)
    want = _conv_tables_expected(d3d, coors_t, num, shp, out, params, max_out)
    for cleared in (False, True):
        _check_conv_tables(_conv_tables(d3d, plug, coors_t, num, shp, max_out, kvol, cleared=cleared), want, max_out)
        plug._workspace.fill_(1)  # nothing of the first build may be needed


@pytest.mark.parametrize("ks,st,pd,dil,tr", CONVS)
@pytest.mark.parametrize("n,room", [(1, 1.0), (30, 1.0), (700, 1.3), (700, 0.4)])
def test_tables_on_the_voxels_of_a_strided_pass(d3d, ks, st, pd, dil, tr, n, room):
    """A second strided kernel and submanifold kernels that look their voxels up where the first kernel has left them."""
    from deploy3d_b200.plugins import SPConvMMPlugin, SubmTables, deserialize_plugin
    shape, cap, first = [2, 13, 24, 67], 750, ((3, 3, 3), (1, 2, 1), ONE, ONE, False)
    coors = np.zeros((cap, 4), np.int32)
    coors[:n] = unique_coors(rng(n), n, shape)
    coors_t, num, shp = _t(coors), torch.tensor([n], dtype=torch.int32, device=DEV), _carrier(shape)
    mid = _out_shape(shape, *first)
    mid_max = max(700, int(_conv_tables_expected(d3d, coors_t, num, shp, mid, first, 1)[0] * room))
    plug = deserialize_plugin("SPConvIdx3d", d3d.data_s_spconv_index(*first[:4], ZERO, mid_max, False, False))
    oc, on, _, _ = _conv_tables(d3d, plug, coors_t, num, shp, mid_max, 27)
    grid = plug.tables_grid(coors_t, num, shp, device=DEV)

    kernels = [(3, 3, 3), (1, 3, 3), (3, 1, 1), (1, 1, 1)]
    for sub in (kernels, kernels[1:3]):
        a, b = ([torch.full((SPConvMMPlugin.table_bytes(int(np.prod(k)), mid_max),), 93, dtype=torch.uint8, device=DEV)
                 for k in sub] for _ in range(2))
        SubmTables(sub).enqueue(oc, on, _carrier(mid), tables=a)
        SubmTables(sub).enqueue(oc, on, _carrier(mid), tables=b, voxel_grid=grid)
        for k, x, y in zip(sub, a, b):
            v = int(np.prod(k))
            assert_tables_equal(table_parts(y, v, mid_max), table_parts(x, v, mid_max), "%s" % (k,))

    params, out = (ks, st, pd, dil, tr), _out_shape(mid, ks, st, pd, dil, tr)
    max_out = max(1, int(_conv_tables_expected(d3d, oc, on, _carrier(mid), out, params, 1)[0] * room))
    want = _conv_tables_expected(d3d, oc, on, _carrier(mid), out, params, max_out)
    second = deserialize_plugin("SPConvIdx3d", d3d.data_s_spconv_index(ks, st, pd, dil, ZERO, max_out, False, tr))
    got = _conv_tables(d3d, second, oc, on, _carrier(mid), max_out, int(np.prod(ks)), voxel_grid=grid, cleared=not tr)
    _check_conv_tables(got, want, max_out)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("n", [1, 400])
def test_subm_tables_cleared_ahead(d3d, grid, n):
    from deploy3d_b200.plugins import SPConvMMPlugin, SubmTables
    shape, cap = GRIDS[grid], 500
    coors = np.zeros((cap, 4), np.int32)
    coors[:n] = unique_coors(rng(n), n, [shape[0], 9, 12, 13])
    coors_t, num = _t(coors), torch.tensor([n], dtype=torch.int32, device=DEV)
    shp = torch.empty([shape[0], 0] + shape[1:], dtype=torch.int32, device=DEV)
    want, got = (torch.full((SPConvMMPlugin.table_bytes(27, cap),), 93, dtype=torch.uint8, device=DEV) for _ in range(2))
    p = SubmTables([(3, 3, 3)])
    p.enqueue(coors_t, num, shp, tables=[want])
    p._workspace.fill_(1)  # nothing of the first build may be needed
    p.clear(coors_t, num, shp, device=torch.device(DEV))
    p.enqueue(coors_t, num, shp, tables=[got], cleared=True)
    assert_tables_equal(table_parts(got, 27, cap), table_parts(want, 27, cap))


@pytest.mark.parametrize("ks,st,pd,dil,tr", [((2, 2, 2), (2, 2, 2), ZERO, ONE, True), ((3, 3, 3), (3, 2, 1), ONE, ONE, True),
                                             ((3, 3, 3), ONE, (1, 1, 16), (1, 1, 16), False)])
def test_conv_tables_cleared_for_a_voxel_grid_they_cannot_walk(d3d, ks, st, pd, dil, tr):
    """Transposed and widely dilated kernels scatter into the forward table although a voxel grid is given: a clear that
    was made without the table, as it is for a voxel grid, is enough all the same."""
    from deploy3d_b200.plugins import deserialize_plugin
    shape, first, n = [2, 13, 24, 67], ((3, 3, 3), (1, 2, 1), ONE, ONE, False), 700
    coors_t, num, shp = _t(unique_coors(rng(n), n, shape)), torch.tensor([n], dtype=torch.int32, device=DEV), _carrier(shape)
    mid = _out_shape(shape, *first)
    mid_max = _conv_tables_expected(d3d, coors_t, num, shp, mid, first, 1)[0]
    plug = deserialize_plugin("SPConvIdx3d", d3d.data_s_spconv_index(*first[:4], ZERO, mid_max, False, False))
    oc, on, _, _ = _conv_tables(d3d, plug, coors_t, num, shp, mid_max, 27)
    grid = plug.tables_grid(coors_t, num, shp, device=DEV)
    params, out = (ks, st, pd, dil, tr), _out_shape(mid, ks, st, pd, dil, tr)
    max_out = _conv_tables_expected(d3d, oc, on, _carrier(mid), out, params, 1)[0]
    want = _conv_tables_expected(d3d, oc, on, _carrier(mid), out, params, max_out)
    second = deserialize_plugin("SPConvIdx3d", d3d.data_s_spconv_index(ks, st, pd, dil, ZERO, max_out, False, tr))
    assert second.tables_ok(oc, on, _carrier(mid))
    for cleared in (False, True):
        got = _conv_tables(d3d, second, oc, on, _carrier(mid), max_out, int(np.prod(ks)), voxel_grid=grid, cleared=cleared)
        _check_conv_tables(got, want, max_out)
        second._workspace.fill_(1)


@pytest.mark.parametrize("words", [0, 1, 2])
def test_output_coordinates_in_an_arena_of_words(d3d, words):
    """Output coordinates that start on any 4 bytes, as a piece of a caller's flat buffer may."""
    from deploy3d_b200.plugins import SPConvMMPlugin, deserialize_plugin
    shape, n = [2, 13, 24, 25], 700
    coors_t, num, shp = _t(unique_coors(rng(n), n, shape)), torch.tensor([n], dtype=torch.int32, device=DEV), _carrier(shape)
    args = (3, 3, 3), (2, 2, 2), ONE, ONE, ZERO, 2000, False, False
    index, num_index, want, on, carrier = d3d.spconv_index(coors_t, num, shp, *args)
    m = int(on.item())
    plug = deserialize_plugin("SPConvIdx3d", d3d.data_s_spconv_index(*args))

    def piece():
        flat = torch.full((4 * 2000 + 4,), -9, dtype=torch.int32, device=DEV)
        return flat, flat[words:words + 8000].view(2000, 4)

    flat, oc = piece()
    plug.enqueue(coors_t, num, shp, outputs=[index, num_index, oc, on, carrier])
    assert torch.equal(oc[:m], want[:m]) and (flat[:words] == -9).all() and (oc[m:] == -9).all()
    flat, oc = piece()
    table = torch.empty(SPConvMMPlugin.table_bytes(27, 2000), dtype=torch.uint8, device=DEV)
    plug.tables(coors_t, num, shp, out_coors=oc, num_act_out=on, table=table)
    key = lambda c: ((c[:, 0] * 7 + c[:, 1]) * 12 + c[:, 2]) * 13 + c[:, 3]
    assert int(on.item()) == m and torch.equal(oc[:m], want[:m][torch.argsort(key(want[:m]))])
    assert (flat[:words] == -9).all() and (oc[m:] == -9).all()


# More blocks than read the counts in front of them for themselves (4096): a scan is launched in between.
def test_conv_numbering_beyond_the_summed_blocks(d3d):
    shape, n, cap = [1, 31, 200, 200], 1060000, 4200 * 256 + 3
    coors = np.zeros((cap, 4), np.int32)
    coors[:n] = unique_coors(rng(9), n, shape)
    args = (3, 1, 1), (2, 1, 1), ZERO, ONE, ZERO
    outs = d3d.spconv_index(_t(coors), torch.tensor([n], dtype=torch.int32, device=DEV), _carrier(shape), *args, 700000, False,
                            False)
    at = coors[:n, None, 1] - np.arange(3)[None]
    ok = (at % 2 == 0) & (at >= 0) & (at // 2 < 15)
    key = (at // 2 * 40000 + (coors[:n, 2] * 200 + coors[:n, 3])[:, None])[ok]
    _, first = np.unique(key, return_index=True)
    want = key[np.sort(first)]
    m = int(outs[3].item())
    got = outs[2].cpu().numpy()[:m]
    assert m == len(want) and (got[:, 1] * 40000 + got[:, 2] * 200 + got[:, 3] == want).all()


def test_conv_tables_beyond_the_summed_blocks(d3d):
    from deploy3d_b200.plugins import deserialize_plugin
    shape, n, max_out = [1, 41, 909, 907], 100000, 220000  # 34 M cells, 4127 blocks of words
    params, out = ((3, 1, 1), ONE, (1, 0, 0), ONE, False), shape
    coors_t, num, shp = _t(unique_coors(rng(4), n, shape)), torch.tensor([n], dtype=torch.int32, device=DEV), _carrier(shape)
    plug = deserialize_plugin("SPConvIdx3d", d3d.data_s_spconv_index(*params[:4], ZERO, max_out, False, False))
    assert plug.tables_ok(coors_t, num, shp)
    got = _conv_tables(d3d, plug, coors_t, num, shp, max_out, 3)
    index, num_index, oc, on, _ = d3d.spconv_index(coors_t, num, shp, *params[:4], ZERO, 600000, False, False)
    m, oc = int(on.item()), oc[:int(on.item())].long()
    order = torch.argsort((oc[:, 1] * out[2] + oc[:, 2]) * out[3] + oc[:, 3])
    ids = torch.empty_like(order)
    ids[order] = torch.arange(m, device=DEV)
    pairs = index[:, :int(num_index.item())].long()
    pairs = pairs[:, pairs[2] >= 0]
    trip = torch.stack([ids[pairs[1]], pairs[2], pairs[0]], 1)
    assert m > max_out
    _check_conv_tables(got, (m, oc[order][:max_out].int(), trip[trip[:, 0] < max_out]), max_out)

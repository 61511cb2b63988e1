"""SPConvMM on the tensor cores at the edges of its units, rounds and accumulators: kernel volumes that leave windows of
offsets and pairs of them half full, tiles shared by the MMA warps, rounds of one to three tiles with a remainder, every
number of accumulators, features, outputs and tables off their boundaries, weights that are not finite, waits that run out.
Held against the SIMT kernel of the same library, which walks the offsets one by one (tests/test_gpu_spconv_tc.py holds both
against the oracle)."""
import ctypes

import numpy as np
import pytest
import torch

from tests._util import assert_feats_close, producer_warps, rng, table_parts, table_row_bits, unique_coors

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _error():
    from deploy3d_b200 import _lib
    code = ctypes.c_int(-1)
    _lib.check("d3d_debug_take_kernel_error", _lib.lib().d3d_debug_take_kernel_error(ctypes.byref(code)))
    return code.value


@pytest.fixture
def wait_limit():
    """Sets the cycles after which a bounded wait gives up; the usual second again afterwards."""
    from deploy3d_b200 import _lib
    set_to = lambda cycles: _lib.check("d3d_debug_set_wait_limit", _lib.lib().d3d_debug_set_wait_limit(cycles))
    yield set_to
    set_to(0)


def _setup(d3d, n, grid, ks, cin, cout, dtype, seed, cap=None, edit=None):
    """Table of a SubM rulebook over n random voxels, features, and a plugin with random weights (`edit` may change them)."""
    from deploy3d_b200.plugins import SPConvMMPlugin, deserialize_plugin
    cap = cap or n
    coors = torch.from_numpy(unique_coors(rng(seed), n, grid)).to(DEV)
    num = torch.tensor([n], dtype=torch.int32, device=DEV)
    outs = d3d.spconv_index(coors, num, torch.empty([grid[0], 0] + grid[1:], dtype=torch.int32, device=DEV), ks, (1,) * 3,
                            tuple(k // 2 for k in ks), (1,) * 3, (0,) * 3, cap, True, False)
    kvol = int(np.prod(ks))
    table = SPConvMMPlugin.prepare(kvol, False, cap, outs[0], outs[1])
    r = rng(seed + 1)
    w = (r.standard_normal((kvol, cin, cout)) * np.sqrt(2.0 / (kvol * cin))).astype(np.float32)
    b = r.standard_normal(cout).astype(np.float32)
    if edit:
        edit(w)
    plug = deserialize_plugin("SPConvMM", d3d.data_s_spconv_mm(ks, cin, cout, cap, True, False, w, b))
    plug.configure(dtype)
    x = torch.from_numpy(r.standard_normal((n, cin)).astype(np.float32)).to(DEV, dtype)
    return plug, x, num, table


def _both(plug, x, num, table, **kw):
    plug.set_kernel(1)
    want = plug.run(x, num, table, **kw).float().cpu().numpy()
    plug.set_kernel(2)
    got = plug.run(x, num, table, **kw)
    assert _error() == 0, "a bounded wait of the tensor-core kernel expired"
    return got, want


@pytest.mark.parametrize("ks", [(1, 1, 1), (3, 1, 1), (5, 1, 1), (1, 3, 3), (5, 3, 1), (3, 3, 3)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 32), (64, 64), (128, 48), (256, 16)])
def test_kernel_volumes(d3d, ks, cin, cout):
    plug, x, num, table = _setup(d3d, 3000, [1, 20, 24, 22], ks, cin, cout, torch.float16, 3)
    got, want = _both(plug, x, num, table, relu=True)
    assert_feats_close(got.float().cpu().numpy(), want, 1e-2, "kernel %s" % (ks,))


@pytest.mark.parametrize("tiles", [1, 2, 147, 149, 297, 445, 593])
@pytest.mark.parametrize("cin,cout", [(32, 64), (64, 128)])
def test_rounds_and_their_remainder(d3d, tiles, cin, cout):
    n = tiles * 128 - 37
    plug, x, num, table = _setup(d3d, n, [2, 40, 48, 44], (3, 1, 3), cin, cout, torch.bfloat16, tiles)
    res = torch.randn((n, cout), device=DEV).bfloat16()
    got, want = _both(plug, x, num, table, relu=True, residual=res)
    assert_feats_close(got.float().cpu().numpy(), want, 1e-2, "%d tiles" % tiles)


@pytest.mark.parametrize("tiles", [148, 296, 297, 443, 444, 445, 593, 900])
@pytest.mark.parametrize("cin,cout", [(32, 32), (64, 64), (128, 64)])
def test_rounds_of_three_tiles(d3d, tiles, cin, cout):
    """Three MMA warps (27 offsets, up to 64 output channels; 64 is the fewest accumulators they run with) over whole rounds and
    remainders, with weights that are held (32 -> 32), streamed and in two parts; a stretch of tiles without an offset, so
    that rounds of one, two and three live tiles follow each other; plain and regrouped."""
    from deploy3d_b200.plugins import SPConvMMPlugin
    n = tiles * 128 - 37
    plug, x, num, table = _setup(d3d, n, [1, 60, 60, 60], (3, 3, 3), cin, cout, torch.bfloat16, tiles)
    _, tile_mask, row_masks, _ = table_parts(table, 27, n)
    gone = torch.zeros(tiles, dtype=torch.bool, device=DEV)
    gone[tiles // 3:tiles // 2] = True
    gone[::7] = True
    gone[1::14] = True
    tile_mask[gone] = 0
    row_masks[gone] = 0
    res = torch.randn((n, cout), device=DEV).bfloat16()
    got, want = _both(plug, x, num, table, residual=res)
    assert_feats_close(got.float().cpu().numpy(), want, 1e-2, "%d tiles" % tiles)
    grouped = SPConvMMPlugin.regroup(27, n, table)
    assert torch.equal(plug.run(x, num, grouped, residual=res), got) and _error() == 0


@pytest.mark.parametrize("cout", [16, 32, 48, 64, 80, 96, 112, 128, 144, 160, 176, 192, 208, 240, 256])
def test_numbers_of_accumulators(d3d, cout):
    """With two and three MMA warps, whose bytes are the same."""
    plug, x, num, table = _setup(d3d, 57000, [2, 40, 48, 44], (3, 1, 1), 32, cout, torch.float16, cout)
    got, want = _both(plug, x, num, table)
    assert_feats_close(got.float().cpu().numpy(), want, 1e-2, "%d output channels" % cout)
    for warps in (16, 24):
        with producer_warps(warps):
            assert torch.equal(plug.run(x, num, table), got) and _error() == 0


@pytest.mark.parametrize("ks", [(3, 3, 3), (3, 1, 1), (5, 1, 3)])
@pytest.mark.parametrize("cin", [16, 32, 64, 128])
@pytest.mark.parametrize("cout", [16, 48, 128, 144, 192, 208])
def test_tile_shared_by_the_mma_warps(d3d, ks, cin, cout):
    """At most one tile to a CTA: the windows of a tile go to the MMA warps in turn.  Tiles that have only even windows, only odd
    ones, a single one, or none; plain and regrouped, whose bytes have to be the same."""
    from deploy3d_b200.plugins import SPConvMMPlugin
    n, kvol = 6 * 128 - 11, int(np.prod(ks))
    plug, x, num, table = _setup(d3d, n, [1, 8, 10, 12], ks, cin, cout, torch.float16, cout + cin)
    _, tile_mask, row_masks, _ = table_parts(table, kvol, n)
    offs = 64 // min(cin, 64)
    window = torch.arange(kvol, device=DEV) // offs
    keep = [window >= 0, window % 2 == 0, window % 2 == 1, window == 1, window < 0, window == 2]
    for t, k in enumerate(keep):
        row_masks[t][~k] = 0
        tile_mask[t] = tile_mask[t] & sum(1 << i for i in range(kvol) if k[i])
    res = torch.randn((n, cout), device=DEV).half()
    got, want = _both(plug, x, num, table, relu=True, residual=res)
    assert_feats_close(got.float().cpu().numpy(), want, 1e-2, "shared tiles")
    grouped = SPConvMMPlugin.regroup(kvol, n, table)
    assert torch.equal(plug.run(x, num, grouped, relu=True, residual=res), got) and _error() == 0


@pytest.mark.parametrize("cin", [16, 32, 64, 128])
def test_features_and_outputs_on_16_bytes(d3d, cin):
    n, cout = 5000, 48
    plug, x, num, table = _setup(d3d, n, [1, 24, 30, 20], (3, 3, 3), cin, cout, torch.float16, 7)
    want = plug.run(x, num, table, relu=True)
    at = lambda t: torch.cat([t.new_zeros(8), t.flatten()])[8:].view(t.shape)
    out = at(torch.zeros_like(want))
    moved = at(x)
    assert moved.data_ptr() % 32 == 16 and out.data_ptr() % 32 == 16
    assert torch.equal(plug.run(moved, num, table, out=out, relu=True), want)
    assert _error() == 0


@pytest.mark.parametrize("ks", [(3, 3, 3), (3, 1, 3)])
@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 48), (32, 96), (64, 64), (64, 80)])
@pytest.mark.parametrize("n", [5000, 30000, 45000])
def test_table_and_features_off_their_boundaries(d3d, n, ks, cin, cout):
    """A table that starts on four bytes (a copy inside a larger buffer), features that start on 16, and both; one tile to a
    CTA, two, and more, which 27 offsets and up to 64 channels run with three MMA warps."""
    plug, x, num, table = _setup(d3d, n, [1, 40, 40, 40], ks, cin, cout, torch.float16, 17)
    want = plug.run(x, num, table, relu=True)
    moved = torch.cat([x.new_zeros(8), x.flatten()])[8:].view(x.shape)
    assert moved.data_ptr() % 32 == 16
    for off in (4, 8, 12):
        buf = torch.empty(table.numel() + 16, dtype=torch.uint8, device=DEV)
        copy = buf[off:off + table.numel()]
        copy.copy_(table)
        assert copy.data_ptr() % 16 == off
        for feats in (x, moved):
            assert torch.equal(plug.run(feats, num, copy, relu=True), want)
    assert torch.equal(plug.run(moved, num, table, relu=True), want) and _error() == 0


@pytest.mark.parametrize("said", [0, 1, 700, 100000])
def test_live_count_only_deals_out_the_tiles(d3d, said):
    """What is computed follows from the table alone."""
    plug, x, num, table = _setup(d3d, 5000, [1, 24, 30, 20], (3, 3, 3), 32, 32, torch.float16, 9, cap=9000)
    want = plug.run(x, num, table)
    got = plug.run(x, torch.tensor([said], dtype=torch.int32, device=DEV), table)
    assert torch.equal(got, want) and _error() == 0


def test_count_that_changes_during_the_launch(d3d):
    """Which CTA computes which tile follows from the table alone: the word of `num_act_out` may be rewritten meanwhile."""
    plug, x, num, table = _setup(d3d, 41000, [2, 40, 48, 44], (3, 1, 3), 32, 32, torch.float16, 13, cap=60000)
    want = plug.run(x, num, table).clone()
    said = num.clone()
    out = torch.empty_like(want)
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(60):
        with torch.cuda.stream(other):
            for v in (0, 100, 41000, 30000, 60000):
                said.fill_(v)
        out.fill_(7.0)
        plug.run(x, said, table, out=out)
    torch.cuda.synchronize()
    assert torch.equal(out, want) and _error() == 0


@pytest.mark.parametrize("empty", ["none", "tail", "middle", "all_but_last", "every_other", "all"])
def test_tiles_without_an_offset(d3d, empty):
    """Tiles no offset feeds, wherever they lie in the table, hold the bias and the residual."""
    cap = 60000
    plug, x, num, table = _setup(d3d, cap, [2, 40, 48, 44], (3, 1, 3), 32, 32, torch.float16, 14)
    _, tile_mask, row_masks, _ = table_parts(table, 9, cap)
    tiles = tile_mask.numel()
    gone = torch.zeros(tiles, dtype=torch.bool, device=DEV)
    gone[{"none": slice(0, 0), "tail": slice(390, tiles), "middle": slice(150, 401), "all_but_last": slice(0, tiles - 1),
          "every_other": slice(0, tiles, 2), "all": slice(0, tiles)}[empty]] = True
    tile_mask[gone] = 0
    row_masks[gone] = 0
    res = torch.randn((cap, 32), device=DEV).half()
    got, want = _both(plug, x, num, table, residual=res)
    assert_feats_close(got.float().cpu().numpy(), want, 1e-2, empty)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e6])
def test_weights_that_are_not_finite(d3d, value):
    """An infinite weight (1e6 is one in fp16) reaches the rows that have an input under its offset and no others."""
    def edit(w):
        w[5, 3, 2] = value
    plug, x, num, table = _setup(d3d, 2000, [1, 24, 30, 20], (3, 3, 3), 32, 32, torch.float16, 11, edit=edit)
    got, want = _both(plug, x, num, table)
    got = got.float().cpu().numpy()
    finite = np.isfinite(want)
    assert 0 < (~finite).sum() < 2000
    np.testing.assert_array_equal(got[~finite], want[~finite])
    # the finite ones: fp32 sums in another order, rounded to fp16 (two kernels; 1e-2 as everywhere between them)
    assert_feats_close(np.where(finite, got, 0), np.where(finite, want, 0), 1e-2, "finite rows")


def test_preceding_kernel_does_not_count_towards_a_wait(d3d, wait_limit):
    """A layer launched while the one in front still runs waits for it without a limit: the bound is on the kernel's own
    hand-overs.  64 voxels with 27 offsets of 256 -> 256 channels are two CTAs of 57 M multiply-adds each on the SIMT kernel, at
    least 440 k cycles at 128 a cycle; the 256 -> 16 layer behind it takes about 40 k in all."""
    first, x, num, table = _setup(d3d, 64, [1, 4, 4, 4], (3, 3, 3), 256, 256, torch.float16, 21)
    second, _, _, _ = _setup(d3d, 64, [1, 4, 4, 4], (3, 3, 3), 256, 16, torch.float16, 22)
    first.set_kernel(1)
    want = second.run(first.run(x, num, table), num, table).clone()
    second.set_dependent_launch(True)
    wait_limit(150000)
    mid, got = torch.empty_like(x), torch.empty_like(want)
    for _ in range(3):
        first.run(x, num, table, out=mid)
        second.run(mid, num, table, out=got)
    assert _error() == 0, "a wait ran out while the preceding kernel was running"
    assert torch.equal(got, want)


@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 64), (64, 64), (64, 128), (256, 256)])
def test_wait_that_gives_up(d3d, wait_limit, cin, cout):
    """A wait that gives up ends the launch with an error word, wherever in the kernel it happens; the launches after it are
    as good as ever."""
    plug, x, num, table = _setup(d3d, 60000, [1, 40, 60, 60], (3, 3, 3), cin, cout, torch.float16, 23)
    want = plug.run(x, num, table, relu=True).clone()
    scrap = torch.empty_like(want)
    codes = set()
    for cycles in (1, 300, 1000, 3000, 10000):
        wait_limit(cycles)
        for _ in range(3):
            plug.run(x, num, table, out=scrap, relu=True)
            codes.add(_error())
    wait_limit(0)
    assert codes - {0}, "no wait gave up"
    for _ in range(3):
        assert torch.equal(plug.run(x, num, table, relu=True), want) and _error() == 0


@pytest.mark.parametrize("ks", [(3, 3, 3), (3, 1, 3)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 32), (64, 64), (64, 128), (128, 48), (256, 256)])
@pytest.mark.parametrize("n", [4000, 20000, 45000])
def test_weights_that_are_not_finite_stay_on_the_tensor_cores(d3d, n, ks, cin, cout):
    """An infinite weight reaches its own output channel in the rows that have an input under its offset, and nothing else:
    the other channels come out with the same bytes as without it, which another kernel's would not."""
    def edit(w):
        w[5, cin - 3, 2] = np.inf

    plain, x, num, table = _setup(d3d, n, [1, 40, 40, 40], ks, cin, cout, torch.bfloat16, 31)
    plug, _, _, _ = _setup(d3d, n, [1, 40, 40, 40], ks, cin, cout, torch.bfloat16, 31, edit=edit)
    res = torch.randn((n, cout), device=DEV).bfloat16()
    want = plain.run(x, num, table, residual=res).float().cpu().numpy()
    got = plug.run(x, num, table, residual=res).float().cpu().numpy()
    assert _error() == 0
    rest = np.arange(cout) != 2
    np.testing.assert_array_equal(got[:, rest], want[:, rest])
    reached = table_row_bits(table_parts(table, int(np.prod(ks)), n)[2])[:, 5, :].reshape(-1)[:n].cpu().numpy()
    np.testing.assert_array_equal(np.isfinite(got[:, 2]), ~reached)
    assert 0 < reached.sum() < n
    np.testing.assert_array_equal(got[~reached, 2], want[~reached, 2])

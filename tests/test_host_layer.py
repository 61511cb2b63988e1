"""What the Python layer decides before any kernel runs: checked without a GPU."""
import pytest
import torch

META = dict(dtype=torch.int32, device="meta")


def _strided(d3d, cap_out=4000):
    from deploy3d_b200.plugins import deserialize_plugin
    return deserialize_plugin("SPConvIdx3d", d3d.data_s_spconv_index((3, 3, 3), (2, 2, 2), (1, 1, 1), (1, 1, 1),
                                                                     (0, 0, 0), cap_out, False, False))


def test_a_device_without_an_index_is_the_current_one(monkeypatch):
    from deploy3d_b200.plugins import cuda_device
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    assert cuda_device("cuda") == cuda_device(torch.device("cuda")) == torch.device("cuda:3")
    assert cuda_device("cuda:1") == torch.device("cuda:1") and cuda_device("cpu") == torch.device("cpu")


def test_what_an_earlier_call_left_is_never_allocated_anew(d3d):
    """A look-up or a cleared grid that does not exist is an error, not fresh memory."""
    from deploy3d_b200.plugins import SubmTables
    plug = _strided(d3d)
    voxels = torch.empty((1000, 4), **META), torch.empty(1, **META), torch.empty((1, 0, 8, 20, 20), **META)
    with pytest.raises(RuntimeError, match="no earlier call"):
        plug.tables_grid(*voxels, device="cuda:0")
    plug._workspace = torch.empty(64, dtype=torch.uint8)  # too small, and on another device
    with pytest.raises(RuntimeError, match="no earlier call"):
        plug.tables_grid(*voxels, device="cuda:0")
    with pytest.raises(RuntimeError, match="no earlier call"):
        plug.tables(*voxels, out_coors=voxels[0], num_act_out=voxels[1], table=voxels[0], cleared=True)
    with pytest.raises(RuntimeError, match="no earlier call"):
        SubmTables([(3, 3, 3)]).enqueue(*voxels, tables=[voxels[0]], cleared=True)


def test_extras_of_the_mean_encoder_keep_their_size():
    """A C caller built against the header passes these 24 bytes; reading past them would take its stack for pointers."""
    import ctypes
    from deploy3d_b200 import _lib
    assert ctypes.sizeof(_lib.MeanEncoderExtras) == 24
    assert [f[0] for f in _lib.MeanEncoderExtras._fields_] == ["lp_feats", "lp_dtype", "lp_channels", "status"]


def _run_python(code):
    """Runs `code` in a fresh process (threads, limits and forks of its own); its output."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, "exit %s\n%s" % (r.returncode, r.stderr[-2000:])
    return r.stdout.split()


def test_compare_where_no_thread_can_start(d3d):
    """The compare of large weights does without its helpers where the process may not have another thread."""
    assert _run_python("""
import resource
import numpy as np
from deploy3d_b200 import _host
same = _host.module().same_bytes
a = np.random.default_rng(1).integers(0, 255, 1 << 20, dtype=np.uint8)
b, c = a.tobytes(), a.copy()
c[-1] ^= 1
now = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (now + (1 << 20), resource.getrlimit(resource.RLIMIT_AS)[1]))  # no room for a stack
print(same(a, b, 0), same(c, b, 0))
""") == ["True", "False"]


@pytest.mark.parametrize("busy", [False, True])
def test_compare_finds_every_difference(d3d, busy):
    """Sizes around the pieces the compare deals out, one byte off anywhere, by several callers at once; `busy`: on one
    core, where helpers are rarely scheduled when they are wanted."""
    out = _run_python("""
import os
import threading
if %r:
    os.sched_setaffinity(0, {next(iter(os.sched_getaffinity(0)))})
import numpy as np
from deploy3d_b200 import _host
same = _host.module().same_bytes
wrong = []
def caller(seed):
    r = np.random.default_rng(seed)
    for n in [1, 262143, 262144, 262145, 327679, 327680, 327681, 1000003] * 10:
        a = r.integers(0, 255, n, dtype=np.uint8)
        b = b"head" + a.tobytes()
        if not same(a, b, 4):
            wrong.append(("equal", n))
        at = int(r.choice([0, n - 1, r.integers(0, n)]))
        a[at] ^= 1
        if same(a, b, 4):
            wrong.append((at, n))
threads = [threading.Thread(target=caller, args=(s,)) for s in range(3)]
[t.start() for t in threads]
[t.join() for t in threads]
print(len(wrong), *wrong[:5])
""" % busy)
    assert out == ["0"]


class _Recorder:
    """Stands in for a plugin object: keeps what it is called with."""

    def __init__(self, name, data_s):
        self.name, self.data_s, self.calls = name, data_s, []

    def enqueue(self, *inputs, **how):
        self.calls.append(inputs)
        return (self,)


@pytest.fixture
def operators(d3d, monkeypatch):
    """The operator layer over recorders, with empty look-ups."""
    from deploy3d_b200.ops import spconv
    monkeypatch.setattr(spconv, "deserialize_plugin", _Recorder)
    monkeypatch.setattr(spconv, "_CACHE", {})
    monkeypatch.setattr(spconv, "_BY_ARGS", {})
    return spconv


def _layer(w, b=None, ksize=(3, 3, 3), cap=10):
    return (None,) * 5 + (ksize, 2, 4, cap, True, False, w, b)


def test_weights_at_many_addresses_are_kept_once(operators):
    import numpy as np
    w = np.random.default_rng(0).standard_normal((27, 2, 4)).astype(np.float32)
    copies = [w.copy() for _ in range(20)]
    plugs = {operators.spconv_mm(*_layer(c)) for c in copies}
    plugs |= {operators.spconv_mm(*_layer(c)) for c in copies}  # found by address now
    assert len(plugs) == 1
    blobs = [v[1] for k, v in operators._BY_ARGS.items() if k[0] == "SPConvMM"]
    assert len(blobs) == 20 and len({id(b) for b in blobs}) == 1


@pytest.mark.parametrize("ksize", [27, [3, 3, 3], (27,), "array"])
def test_kernel_size_in_any_form(operators, ksize):
    """The blob holds the kernel volume only, so a number does for kernel_size as well as extents in any container."""
    import numpy as np
    w = np.ones((27, 2, 4), np.float32)
    form = np.array([3, 3, 3]) if ksize == "array" else ksize
    for _ in range(2):
        assert operators.spconv_mm(*_layer(w, ksize=form)) is operators.spconv_mm(*_layer(w))


def test_arguments_that_change_in_place(operators):
    """A size held in a tensor is read on every call, as a number would be."""
    import numpy as np
    rows = torch.tensor(10)
    k, one = (3, 3, 3), (1, 1, 1)
    w = np.ones((27, 2, 4), np.float32)
    for n in (10, 25, 10):
        rows.fill_(n)
        plug = operators._plugin_by_args("SPConvIdx3d", (k, one, one, one, (0, 0, 0), rows, True, False),
                                         operators.data_s_spconv_index)
        assert plug.data_s == operators.data_s_spconv_index(k, one, one, one, (0, 0, 0), n, True, False)
        plug = operators.spconv_mm(*_layer(w, cap=rows))
        assert plug.data_s == operators.data_s_spconv_mm(k, 2, 4, n, True, False, w)
    assert all(operators._plain(key) for key in operators._BY_ARGS)


def test_tables_ask_for_what_they_use(d3d):
    """Strided tables: 8 bytes per 32 cells and a count per 8192 of them; submanifold tables: their look-up.  Not the grid
    and the pair lists of a rulebook."""
    import ctypes
    from deploy3d_b200 import _lib
    from deploy3d_b200.plugins import SPConvIdxPlugin, _desc_of
    for shape, n in (([1, 41, 1440, 1440], 300000), ([1, 21, 720, 720], 500000), ([2, 5, 9, 11], 64)):
        descs = [_desc_of(t) for t in (torch.empty((n, 4), **META), torch.empty(1, **META),
                                       torch.empty(shape[:1] + [0] + shape[1:], **META))]
        plug = _strided(d3d)
        out = [shape[0]] + [(e - 1) // 2 + 1 for e in shape[1:]]
        cells = out[0] * out[1] * out[2] * out[3]
        nbytes = plug._tables_workspace_size(descs)
        assert cells // 4 <= nbytes <= cells // 4 + cells // 2048 + 1024 < plug.workspace_size(descs)
        size = ctypes.c_size_t(0)
        _lib.check("workspace", _lib.lib().d3d_spconv_subm_tables_workspace(_lib.desc_array(descs), 3, ctypes.byref(size)))
        cells = shape[0] * shape[1] * shape[2] * shape[3]
        if cells <= 64 * n:
            assert cells * 4 <= size.value <= cells * 4 + 256
        else:  # a bit per cell and hash slots for four to eight times the rows
            assert size.value <= cells // 8 + 64 * n + 1024
    far = [_desc_of(t) for t in (torch.empty((8, 4), **META), torch.empty(1, **META), torch.empty((1, 0, 41, 800, 800), **META))]
    assert not SPConvIdxPlugin.tables_ok(plug, torch.empty((8, 4), **META), torch.empty(1, **META),
                                         torch.empty((1, 0, 41, 800, 800), **META))
    with pytest.raises(_lib.D3DError):
        plug._tables_workspace_size(far)

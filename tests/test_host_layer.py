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

"""``spconv_index``, ``spconv_mm``, ``bev_densify`` (deploy3d/symfun/ops/spconv/*.py)."""
import numpy as np

from .. import _host
from ..plugins import deserialize_plugin

_CACHE = {}
# Plugins found by the arguments of an operator call instead of by their serialized form: the blob of a large layer is
# megabytes that would be put together and hashed on every call.
_BY_ARGS = {}
_BLOB_HEADER = 19  # bytes of an SPConvMM blob before the weights


def _plugin(name, data_s):
    return _plugin_and_blob(name, data_s)[0]


def _plugin_and_blob(name, data_s):
    """The plugin and the one copy of its blob that is kept, however many equal ones are passed."""
    key = (name, data_s)
    found = _CACHE.get(key)
    if found is None:
        if len(_CACHE) > 256:
            _CACHE.clear()
            _BY_ARGS.clear()
        found = _CACHE[key] = (deserialize_plugin(name, data_s), data_s)
    return found


def _plain(v):
    """Whether equal keys mean equal values for good: numbers and tuples of them, not tensors (equal to themselves whatever
    they hold by now)."""
    return v is None or isinstance(v, (int, float, str, np.generic)) or (type(v) is tuple and all(map(_plain, v)))


def _volume(kernel_size):
    """Kernel volume of extents in any container, or of the volume itself."""
    try:
        v = 1
        for k in kernel_size:
            v *= int(k)
        return v
    except TypeError:
        return int(kernel_size)


def _plugin_by_args(name, args, data_s):
    """The plugin `name` whose blob is data_s(*args); kept for arguments that determine the blob."""
    key = (name,) + args
    try:
        plug = _BY_ARGS.get(key)
    except TypeError:  # lists or arrays where the operator is documented with tuples
        return _plugin(name, data_s(*args))
    if plug is None:
        plug = _plugin(name, data_s(*args))
        if _plain(key):
            if len(_BY_ARGS) > 1024:
                _BY_ARGS.clear()
            _BY_ARGS[key] = plug
    return plug


def data_s_spconv_index(kernel_size, stride, padding, dilation, out_padding, max_num_act_out, subm, transpose):
    """Blob of SPConvIdx{N}d (deploy3d/symfun/ops/spconv/spconv_index.py:94-101; trt/spconv/index_trt.cu:39-50)."""
    data = np.array(kernel_size, dtype=np.int32).tobytes()
    data += np.array(stride, dtype=np.int32).tobytes()
    data += np.array(padding, dtype=np.int32).tobytes()
    data += np.array(dilation, dtype=np.int32).tobytes()
    data += np.array(out_padding, dtype=np.int32).tobytes()
    data += np.array([max_num_act_out], dtype=np.int32).tobytes()
    data += np.array([subm], dtype=np.bool_).tobytes()
    data += np.array([transpose], dtype=np.bool_).tobytes()
    return data


def spconv_index(in_coors, num_act_in, in_spatial_shape, kernel_size, stride, padding, dilation, out_padding,
                 max_num_act_out, subm, transpose):
    """Returns (index, num_index) when ``subm`` else (index, num_index, out_coors, num_act_out, out_spatial_shape).

    in_coors int32 [maxNumActIn, NDim+1]; num_act_in int32 [1]; in_spatial_shape: zero-element tensor
    [B, 0, D0, ..] whose *shape* carries the grid extent (deploy3d/symfun/ops/spconv/spconv_index.py:8-21)."""
    plug = _plugin_by_args("SPConvIdx%dd" % (in_coors.shape[1] - 1),
                           (kernel_size, stride, padding, dilation, out_padding, max_num_act_out, subm, transpose),
                           data_s_spconv_index)
    return plug.enqueue(in_coors, num_act_in, in_spatial_shape)


def data_s_spconv_mm(kernel_size, in_channels, out_channels, max_num_act_out, subm, inverse, weight, bias=None):
    """Blob of SPConvMM (deploy3d/symfun/ops/spconv/spconv_mm.py:54-63; trt/spconv/mm_trt.cu:27-37)."""
    data = np.array([int(np.prod(kernel_size))], dtype=np.int32).tobytes()
    data += np.array([in_channels], dtype=np.int32).tobytes()
    data += np.array([out_channels], dtype=np.int32).tobytes()
    data += np.array([max_num_act_out], dtype=np.int32).tobytes()
    data += np.array([subm], dtype=np.bool_).tobytes()
    data += np.array([inverse], dtype=np.bool_).tobytes()
    data += np.array([bias is not None], dtype=np.bool_).tobytes()
    data += np.ascontiguousarray(weight, dtype=np.float32).tobytes()
    if bias is not None:
        data += np.ascontiguousarray(bias, dtype=np.float32).tobytes()
    return data


def spconv_mm(in_feats, num_act_in, num_act_out, index, num_index, kernel_size, in_channels, out_channels,
              max_num_act_out, subm, inverse, weight, bias=None):
    """out_feats [maxNumActOut, Cout] in the dtype of in_feats (float16, bfloat16 or float32).

    weight: numpy [kVol, Cin, Cout] (flattened is accepted), bias: numpy [Cout] or None
    (deploy3d/symfun/ops/spconv/spconv_mm.py:21-35)."""
    inputs = (in_feats, num_act_in, num_act_out, index, num_index)
    # The plugin that these very arrays made last time is launched at once, and while the GPU works the arrays are
    # compared with the weights it holds, byte by byte: arrays whose contents changed since then (or another array at
    # the same address) get a plugin of their own, whose launch overwrites the first one's output.
    key = None
    if type(weight) is np.ndarray and weight.dtype == np.float32 and weight.flags.c_contiguous and (
            bias is None or (type(bias) is np.ndarray and bias.dtype == np.float32 and bias.flags.c_contiguous)):
        key = ("SPConvMM", _volume(kernel_size), in_channels, out_channels, max_num_act_out, bool(subm), bool(inverse),
               weight.ctypes.data, weight.nbytes, None if bias is None else bias.nbytes)
        found = _BY_ARGS.get(key)
        if found is not None:
            plug, blob = found
            out = plug.enqueue(*inputs)[0]
            same = _host.module().same_bytes
            end = _BLOB_HEADER + weight.nbytes
            if same(weight, blob, _BLOB_HEADER) and (bias is None or same(bias, blob, end)):
                return out
    data = data_s_spconv_mm(kernel_size, in_channels, out_channels, max_num_act_out, subm, inverse, weight, bias)
    found = _plugin_and_blob("SPConvMM", data)
    if key is not None and _plain(key):
        if len(_BY_ARGS) > 1024:
            _BY_ARGS.clear()
        _BY_ARGS[key] = found
    return found[0].enqueue(*inputs)[0]


def data_s_bev_densify(out_channels):
    return np.array([out_channels], dtype=np.int32).tobytes()


def bev_densify(in_feats, in_coors, num_act_in, in_spatial_shape, out_channels):
    """Dense [B, C*Z, Y, X] map (deploy3d/symfun/ops/spconv/bev_densify.py:18-28)."""
    plug = _plugin_by_args("BEVDensify", (out_channels,), data_s_bev_densify)
    return plug.enqueue(in_feats, in_coors, num_act_in, in_spatial_shape)[0]

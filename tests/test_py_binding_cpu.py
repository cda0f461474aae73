"""The CPython binding (lib/_kpx_py.<abi>.so) converts what the ctypes signatures convert and refuses what
they refuse; no GPU is needed: the entry points check their arguments before they touch a device."""

import ctypes

import numpy as np
import pytest

from orinmllm_b200 import capi


@pytest.fixture()
def entries(native_libs):
    module = capi._entries()
    module.set_stream_source(lambda: 0, lambda device: 0)
    yield module
    module.set_stream_source(capi._current_device, capi._raw_stream)


def _decode(**change):
    t = np.zeros(64, np.float32)
    args = dict(out=t, q=t, k_pool=t, v_pool=t, layout=capi.layout_paged(capi.KPX_F32, 2), block_table=t,
                max_blocks_per_seq=1, seq_lens=t, len_bias=0, batch=0, num_q_heads=2, scale=1.0, workspace=1 << 20,
                workspace_bytes=1 << 40)
    args.update(change)
    capi.paged_decode(**args)


class _Tensor:
    def __init__(self, address):
        self.address = address

    def data_ptr(self):
        return self.address


def test_accepted(entries):
    _decode()  # a batch of 0 is done without a device
    _decode(out=4096, q=_Tensor(8192), scale=2, stream=np.int64(0))
    _decode(batch=1 << 32)  # integers are cut to their width, as ctypes cuts them
    _decode(workspace=_Tensor(256), block_table=None)


class _Holder:
    def __init__(self, value):
        self._as_parameter_ = value


def test_ctypes_scalars(entries):
    """A scalar of the argument's own ctypes type is the number it holds."""
    _decode(batch=ctypes.c_int32(0), scale=ctypes.c_float(0.5), max_blocks_per_seq=_Holder(1), len_bias=_Holder(ctypes.c_int32(0)),
            workspace_bytes=ctypes.c_int64(1 << 40))
    with pytest.raises(capi.KpxError) as e:
        _decode(workspace_bytes=ctypes.c_int64(16))
    assert e.value.status == capi.KPX_ERR_WORKSPACE_TOO_SMALL
    for change in (dict(batch=ctypes.c_int64(0)), dict(batch=ctypes.c_float(0)), dict(scale=ctypes.c_double(1)),
                   dict(batch=_Holder("0")), dict(scale=_Holder("1"))):
        with pytest.raises(TypeError):
            _decode(**change)


@pytest.mark.parametrize("change", [dict(max_blocks_per_seq=1.0), dict(q="text"), dict(q=b"bytes"), dict(layout=None),
                                    dict(layout=b"short"), dict(scale="1"), dict(batch=None), dict(q=_Tensor("x")),
                                    dict(batch=np.int64(0))])
def test_refused_before_the_call(entries, change):
    with pytest.raises(TypeError):
        _decode(**change)


class _Other(ctypes.Structure):
    _fields_ = capi.KvLayout._fields_


class _Longer(capi.KvLayout):
    _fields_ = [("note", ctypes.c_int64)]


@pytest.mark.parametrize("layout", [bytes(bytearray(ctypes.sizeof(capi.KvLayout))), _Other(), (ctypes.c_int64 * 6)(),
                                    np.zeros(6, np.int64)], ids=["bytes", "structure", "array", "numpy"])
def test_only_a_layout_is_a_layout(entries, layout):
    """Memory of the layout's size, with a layout's contents even, is not taken for one."""
    assert memoryview(layout).nbytes == ctypes.sizeof(capi.KvLayout)
    if isinstance(layout, ctypes.Structure):
        ctypes.memmove(ctypes.byref(layout), ctypes.byref(capi.layout_paged(capi.KPX_F32, 2)), ctypes.sizeof(layout))
    with pytest.raises(TypeError):
        _decode(layout=layout)
    longer = _Longer()
    ctypes.memmove(ctypes.byref(longer), ctypes.byref(capi.layout_paged(capi.KPX_F32, 2)), ctypes.sizeof(capi.KvLayout))
    _decode(layout=longer)  # a type derived from it is one


def test_status_becomes_an_error(entries):
    with pytest.raises(capi.KpxError) as e:
        _decode(out=None)
    assert e.value.status == capi.KPX_ERR_INVALID_ARGUMENT
    with pytest.raises(capi.KpxError) as e:
        _decode(q=8)  # not 16-byte aligned: the address arrived as it is
    assert e.value.status == capi.KPX_ERR_INVALID_ARGUMENT
    with pytest.raises(capi.KpxError) as e:
        _decode(workspace_bytes=16)
    assert e.value.status == capi.KPX_ERR_WORKSPACE_TOO_SMALL


def test_views_of_arrays_keep_their_address(entries):
    t = np.zeros(64, np.float32)
    first = 1 if t.ctypes.data % 16 == 0 else (16 - t.ctypes.data % 16) // 4 + 1
    with pytest.raises(capi.KpxError):
        _decode(q=t[first:])      # off a 16-byte boundary
    _decode(q=t[first - 1::4])    # on one, strided


def test_number_of_arguments(entries):
    with pytest.raises(TypeError):
        entries.paged_decode(1, 2, 3)


def test_the_file_is_this_interpreters(native_libs, monkeypatch, tmp_path):
    """The extension's name carries the interpreter's ABI, another interpreter's file is not loaded in
    its place, and without Python.h everything else is built."""
    import sysconfig
    from orinmllm_b200 import build
    assert build.py_binding().exists()
    assert build.py_binding().name == "_kpx_py" + sysconfig.get_config_var("EXT_SUFFIX") != "_kpx_py.so"
    monkeypatch.setattr(capi, "_py", None)
    monkeypatch.setattr(capi, "LIB_DIR", tmp_path)
    monkeypatch.setattr(capi, "lib", lambda: None)
    for name in ("_kpx_py.so", "_kpx_py.cpython-399-x86_64-linux-gnu.so"):
        (tmp_path / name).symlink_to(build.py_binding())
    with pytest.raises(RuntimeError, match="build the native libraries"):
        capi._entries()
    monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    assert build.build_py(force=True) is None

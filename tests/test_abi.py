"""The C-ABI library loads without a GPU and exports every symbol the public header declares."""
import ctypes
import os
import re

import pytest

from cuda_mace_b200 import _abi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "cuda_mace_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(cmace_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported(built_library):
    lib = ctypes.CDLL(built_library)
    names = declared_symbols()
    assert len(names) >= 35
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing, f"declared in include/cuda_mace_b200.h but not exported: {missing}"


def test_binding_covers_header(built_library):
    names = set(declared_symbols()) - {"cmace_last_error"}
    assert names == set(_abi.SIGNATURES), names ^ set(_abi.SIGNATURES)


def test_version_and_queries_need_no_gpu(built_library):
    assert _abi.call("cmace_abi_version") == 1
    # pure host arithmetic: chunking rule of the backward scratch
    assert _abi.call("cmace_imp_bwd_scratch_elems", 1000, 128, 0) == 0       # f32, one 128-channel chunk
    assert _abi.call("cmace_imp_bwd_scratch_elems", 1000, 128, 1) == 2 * 16 * 1000  # f64, two chunks
    assert _abi.call("cmace_imp_bwd_scratch_elems", 1000, 96, 0) == 3 * 16 * 1000   # f32, three 32-channel chunks


def test_fused_layout_of_earlier_callers_is_not_read(built_library):
    """A caller that lays fused_w_back out as earlier libraries read it leaves the word after fused_scale 0: its second layer
    writes the radial weights, which the workspace then has room for."""
    header = open(os.path.join(ROOT, "include", "cuda_mace_b200.h")).read()
    assert int(re.search(r"#define CMACE_FUSED_LAYOUT (\d+)", header).group(1)) == _abi.FUSED_LAYOUT
    m = _abi.StepModel(channels=128, elements=2, nbessel=8, fused_w=1, fused_w_back=1, fused_layout=_abi.FUSED_LAYOUT)
    E = 1024
    size = lambda: _abi.call("cmace_step_workspace_bytes", ctypes.byref(m), 10, 10, E)
    fused = size()
    m.fused_layout = 0
    assert size() == fused + E * 4 * 128 * 4


@pytest.mark.parametrize("channels", [32, 64, 96])
def test_fused_layout_of_narrow_models_has_a_name_of_its_own(built_library, channels):
    """As above: neither no name nor the one of 128 channels makes the library read what a narrow model's arrays hold, nor the
    other way round."""
    header = open(os.path.join(ROOT, "include", "cuda_mace_b200.h")).read()
    assert int(re.search(r"#define CMACE_FUSED_LAYOUT_NARROW (\d+)", header).group(1)) == _abi.FUSED_LAYOUT_NARROW
    E = 1024

    def size(C, layout):
        m = _abi.StepModel(channels=C, elements=2, nbessel=8, fused_w=1, fused_w_back=1, fused_layout=layout)
        return _abi.call("cmace_step_workspace_bytes", ctypes.byref(m), 10, 10, E)

    fused = size(channels, _abi.FUSED_LAYOUT_NARROW)
    for layout in (0, 1, _abi.FUSED_LAYOUT):
        assert size(channels, layout) == fused + E * 4 * channels * 4
    assert size(128, _abi.FUSED_LAYOUT_NARROW) == size(128, 0)


def test_argument_errors_are_reported_not_raised(built_library):
    lib = _abi.load()
    rc = lib.cmace_imp_fwd_f32(None, None, None, None, None, 4, 4, 33, None, None)
    assert rc == 3  # CMACE_ERR_UNSUPPORTED: channels not a multiple of 32
    assert b"multiple of 32" in lib.cmace_last_error()
    rc = lib.cmace_linear_f32(None, None, None, None, 1, 5, 32, 32, 1.0, None, None)
    assert rc == 1 and b"null" in lib.cmace_last_error()

"""The C-ABI library loads and exports every symbol ``include/analog_b200.h`` declares
(no compute calls: this runs without a GPU)."""
import ctypes
import os
import re

import pytest

from aihwkit_lightning_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "analog_b200.h")


def declared_functions():
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(al_[a-z0-9_]+)\s*\(", text)))


def test_header_and_binding_agree():
    assert declared_functions() == sorted(_lib.SYMBOLS)


def test_library_exports_every_symbol():
    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip("library not built (python aihwkit-lightning_b200/build.py)")
    lib = ctypes.CDLL(_lib.LIB_PATH)
    for name in declared_functions():
        assert hasattr(lib, name), name
    lib.al_version.restype = ctypes.c_int32
    assert lib.al_version() >= 1
    lib.al_status_str.restype = ctypes.c_char_p
    assert lib.al_status_str(0) == b"ok"
    assert b"timed out" in lib.al_status_str(4)


def test_struct_sizes_match_the_header():
    """AlDesc mixes int32 and double fields: the ctypes mirror must agree with the C layout."""
    import subprocess
    import tempfile

    src = '#include "analog_b200.h"\n#include <stdio.h>\nint main(){printf("%zu %zu %zu\\n", sizeof(AlDesc), sizeof(AlForwardArgs), sizeof(AlBackwardArgs));return 0;}\n'
    with tempfile.TemporaryDirectory() as tmp:
        c_file = os.path.join(tmp, "s.c")
        open(c_file, "w").write(src)
        exe = os.path.join(tmp, "s")
        subprocess.check_call(["gcc", "-I", os.path.join(ROOT, "include"), c_file, "-o", exe])
        sizes = [int(v) for v in subprocess.check_output([exe]).split()]
    assert sizes == [ctypes.sizeof(_lib.AlDesc), ctypes.sizeof(_lib.AlForwardArgs),
                     ctypes.sizeof(_lib.AlBackwardArgs)]


def test_bad_arguments_are_rejected_without_a_gpu():
    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip("library not built")
    lib = _lib.load()
    assert lib.al_forward(None, None, None) == _lib.AL_ERR_BAD_ARGUMENT
    desc = _lib.AlDesc()
    desc.M, desc.K, desc.N, desc.T = 4, 8, 4, 1
    desc.dtype = 7
    args = _lib.AlForwardArgs()
    assert lib.al_forward(desc, args, None) == _lib.AL_ERR_BAD_ARGUMENT
    desc.dtype = 0
    desc.inp_res = 254.0  # DAC without an input range
    assert lib.al_forward(desc, args, None) == _lib.AL_ERR_BAD_ARGUMENT
    assert b"input range" in lib.al_last_error()
    desc.inp_res = -1.0
    ends = (ctypes.c_int32 * 1)(7)  # last end != K
    args.tile_ends = ends
    assert lib.al_forward(desc, args, None) == _lib.AL_ERR_BAD_ARGUMENT
    with pytest.raises(AssertionError):
        _lib.check(_lib.AL_ERR_BAD_ARGUMENT)


def test_descriptor_has_the_layout_of_version_1():
    """A caller built against the first header passes 148 bytes of fields and 4 of padding that it never wrote: nothing
    of the call may depend on those."""
    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip("library not built")
    lib = _lib.load()
    assert _lib.AlDesc.save_for_backward.offset == 144 and ctypes.sizeof(_lib.AlDesc) == 152
    raw = (ctypes.c_ubyte * 152)()
    desc = _lib.AlDesc.from_buffer(raw)
    desc.M, desc.K, desc.N, desc.T = 4, 16, 8, 2
    desc.dtype, desc.ir_mode, desc.inp_res = 1, 1, 254.0
    args = _lib.AlForwardArgs()
    args.x = args.w = args.out = 256
    args.tile_ends = _lib.tile_ends_array([8, 8])
    for fill in (0x00, 0xAB):
        raw[148:152] = [fill] * 4
        assert lib.al_forward(desc, args, None) == _lib.AL_ERR_BAD_ARGUMENT  # refused on the host: no ranges given
        assert b"static input range needs input_range" in lib.al_last_error(), fill


def test_uses_tcgen05_speaks_for_the_engine_of_the_descriptor():
    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip("library not built")
    lib = _lib.load()
    desc = _lib.AlDesc()
    desc.M, desc.K, desc.N, desc.T = 64, 1000, 777, 2
    desc.dtype, desc.ir_mode, desc.inp_res = 1, 2, 254.0
    ends = _lib.tile_ends_array([500, 500])
    assert lib.al_operand_pitch(desc, ends) == 1008
    assert lib.al_uses_tcgen05(desc, ends) == 0  # dense operands: CUDA cores
    desc.engine = _lib.AL_ENGINE_PITCHED
    assert lib.al_uses_tcgen05(desc, ends) == 1
    desc.N, desc.K = 776, 1008
    assert lib.al_uses_tcgen05(desc, _lib.tile_ends_array([504, 504])) == 0  # no pitched layout to announce

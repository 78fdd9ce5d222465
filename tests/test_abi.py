"""CPU: the C-ABI library builds, loads, and exports every symbol include/rotor_b200.h declares.
No compute call is made here (there is no GPU)."""
import ctypes
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "rotor_b200.h")
LIB = os.path.join(ROOT, "rotor-rag_b200", "rotor_b200", "librotor_b200.so")


def declared_functions():
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    text = re.sub(r"^\s*#.*$", "", text, flags=re.M)          # preprocessor lines are not declarations
    return sorted(set(re.findall(r"\b([A-Za-z_][A-Za-z0-9_]*)\s*\([^;{]*\)\s*;", text)))


@pytest.fixture(scope="module")
def lib():
    if not os.path.exists(LIB):
        subprocess.check_call(["make", "-s", "-C", os.path.join(ROOT, "rotor-rag_b200", "csrc")])
    return ctypes.CDLL(LIB)


def test_header_declares_functions():
    names = declared_functions()
    assert "rotor_b200_bitlinear_acc" in names and "bitnet_to_rotor" in names
    assert len(names) >= 20


def test_every_declared_symbol_is_exported(lib):
    missing = [n for n in declared_functions() if not hasattr(lib, n)]
    assert not missing, f"declared in the header but not exported: {missing}"


def test_python_binding_matches_header():
    from rotor_b200 import abi
    bound = set(abi._SIGNATURES)
    declared = set(declared_functions())
    assert declared <= bound, f"header functions without a ctypes signature: {sorted(declared - bound)}"
    assert bound <= declared, f"ctypes signatures without a header declaration: {sorted(bound - declared)}"


def test_pure_host_queries(lib):
    lib.rotor_b200_tiles_bytes.restype = ctypes.c_size_t
    lib.rotor_b200_tiles_bytes.argtypes = [ctypes.c_size_t, ctypes.c_size_t]
    assert lib.rotor_b200_tiles_bytes(6912, 2560) == 6912 * 2560 // 4
    assert lib.rotor_b200_tiles_bytes(20, 72) == 32 * 128 // 4      # padded to 32 x 128
    lib.rotor_b200_status_string.restype = ctypes.c_char_p
    assert lib.rotor_b200_status_string(0) == b"ok"
    assert lib.rotor_b200_version() >= 100


def test_argument_errors_do_not_need_a_gpu(lib):
    # null pointers and zero sizes are rejected before any CUDA call
    lib.rotor_b200_bitlinear_acc.restype = ctypes.c_int
    lib.rotor_b200_bitlinear_acc.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_size_t, ctypes.c_void_p,
                                             ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_int,
                                             ctypes.c_void_p]
    assert lib.rotor_b200_bitlinear_acc(None, 16, 128, None, None, 1, None, 0, None) == 1
    lib.rotor_b200_pack.restype = ctypes.c_int
    lib.rotor_b200_pack.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_void_p]
    assert lib.rotor_b200_pack(None, None, 6, None, None) == 1      # length must be a multiple of 4


@pytest.mark.parametrize("out,inn", [(0, 128), (16, 0), (0, 0)])
@pytest.mark.parametrize("rows,terms,variant", [(1, 1, 0), (4, 2, 0), (5, 3, 0), (1, 1, 2)])
def test_layer_call_of_no_rows_or_columns_is_an_argument_error(lib, out, inn, rows, terms, variant):
    """A weight matrix of size zero is refused on the host, before a grid is sized by it and before any CUDA call (the
    addresses are never read: one call in a process of its own, which a division by zero would end)."""
    import sys
    code = """
import ctypes as C, sys
f = C.CDLL(sys.argv[1]).rotor_b200_bitlinear_forward
f.argtypes = [C.c_void_p, C.c_size_t, C.c_size_t, C.c_void_p, C.c_size_t, C.c_int, C.c_float, C.c_void_p, C.c_void_p, C.c_void_p,
              C.c_size_t, C.c_int, C.c_void_p]
out, inn, rows, terms, variant = map(int, sys.argv[2:])
print(f(1 << 20, out, inn, 1 << 21, rows, terms, 1.0, None, 1 << 22, 1 << 23, 1 << 20, variant, None))
"""
    r = subprocess.run([sys.executable, "-c", code, LIB] + [str(v) for v in (out, inn, rows, terms, variant)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.split() == ["1"], (r.returncode, r.stdout, r.stderr)


def test_stream_without_the_short_cut():
    """A torch without the private entry gives the same address through the public one."""
    from types import SimpleNamespace
    from rotor_b200 import abi
    cuda = SimpleNamespace(current_stream=lambda device: SimpleNamespace(cuda_stream=100 + device))
    assert abi._stream_lookup(SimpleNamespace(_C=SimpleNamespace(), cuda=cuda))(3) == 103
    short = SimpleNamespace(_C=SimpleNamespace(_cuda_getCurrentRawStream=lambda device: 200 + device), cuda=cuda)
    assert abi._stream_lookup(short)(3) == 203

"""The keys of the j-side list (rockable_gb300/csrc/rk_jkey.cuh), compiled for
the host: entries keep their index, and bodies order above them, up to the
longest list and the largest body index."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include "rk_jkey.cuh"
extern "C" uint64_t key(int j, long e) { return rk::jkey(j, e); }
extern "C" int entry(uint64_t k) { return rk::jkey_entry(k); }
extern "C" int body_bit() { return rk::kJkeyBody; }
extern "C" long most() { return rk::kMaxEntries; }
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("jkey")
    src, so = d / "jkey.cpp", d / "jkey.so"
    src.write_text(SRC)
    subprocess.check_call(["g++", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "rockable_gb300", "csrc"),
                           str(src), "-o", str(so)])
    L = ctypes.CDLL(str(so))
    L.key.argtypes, L.key.restype = [ctypes.c_int, ctypes.c_long], ctypes.c_uint64
    L.entry.argtypes = [ctypes.c_uint64]
    L.most.restype = ctypes.c_long
    return L


def test_keys_hold_every_entry_and_body(lib):
    most = lib.most()
    assert most == 2 ** 31 - 1
    entries = [0, 1, 2 ** 27 - 1, 2 ** 27, 2 ** 28 + 5, most - 1]
    bodies = [0, 1, 50000, 2 ** 21 - 2, 2 ** 21 - 1]
    keys = [lib.key(j, e) for j in bodies for e in entries]
    assert keys == sorted(set(keys))
    assert [lib.entry(k) for k in keys] == entries * len(bodies)
    assert [k >> lib.body_bit() for k in keys] == [j for j in bodies for _ in entries]
    assert keys[-1] < 2 ** (lib.body_bit() + 21)

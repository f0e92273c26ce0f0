"""Launches that opt in to large shared memory or large clusters do so on every device they run on:
the library's host code over a runtime that refuses what the current device has not allowed
(fake_cudart.cpp), first on one device, then on another.  CPU only; no kernel runs."""
import ctypes
import glob
import importlib
import os
import subprocess

import pytest

from conftest import ROOT

CUDA = "/usr/local/cuda/include"
if not os.path.exists(os.path.join(CUDA, "cuda_runtime_api.h")):
    pytest.skip("needs the CUDA headers", allow_module_level=True)


@pytest.fixture(scope="module")
def host(me, tmp_path_factory):
    lib = me._lib
    importlib.import_module("motion_engine_b200.build").build()
    so = str(tmp_path_factory.mktemp("fake") / "libb2c_fake.so")
    objects = sorted(glob.glob(os.path.join(os.path.dirname(lib.__file__), "_build", "*.o")))
    # -Bsymbolic: the library's calls go to the fake, whatever runtime the process has loaded
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CUDA, "-o", so,
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), *objects], check=True)
    L = ctypes.CDLL(so, mode=os.RTLD_LAZY)  # calls that no launch path makes stay unresolved
    for name, (args, res) in lib._SIGS.items():
        f = getattr(L, name)
        f.argtypes, f.restype = args, res
    return lib, L


_room = ctypes.create_string_buffer(1 << 16)


def _filled(S, **values):
    """A struct whose pointers are not NULL (nothing follows them) and whose other fields are given."""
    s = S()
    for name, t in S._fields_:
        if t is ctypes.c_void_p:
            setattr(s, name, ctypes.addressof(_room))
    for name, v in values.items():
        setattr(s, name, v)
    return s


N = 20000
ROW, FIXED, FIRST, ISLANDS = 64, 1, 32, 256


def _solve(lib, L, blocks, flags, n):
    p = _filled(lib.ColorParams, vit=4, pit=2, max_points=8, flags=flags, mu=0.5, t2d=1.0, color_cap=512,
                solve_blocks=blocks, barrier_timeout_ns=0, body_mu=None)
    b = _filled(lib.Bodies, n=n)
    kept = _filled(lib.Contacts, capacity=8 * n)
    pr = _filled(lib.Pairs, capacity=4 * n, max_colors=512, kslots=8, n_scenes=7)
    hdr = ctypes.addressof(_room)
    B = ctypes.byref
    rc = L.b2c_color_pairs(B(b), B(pr), hdr, B(p), None)
    return rc or L.b2c_color_solve(B(b), B(kept), B(pr), hdr, B(p), 0.004, None)


def _ncp(lib, L, dtype, blocks):
    sc = _filled(lib.NcpScene, dtype=dtype, n_c=4 * N, n_b=N)
    st = _filled(lib.NcpState, n_bodies=N, max_contacts=4 * N, max_colors=1024)
    p = _filled(lib.NcpParams, desaxce=1, solve_blocks=blocks)
    B, q = ctypes.byref, ctypes.addressof(_room)
    rc = L.b2c_ncp_color(B(sc), B(st), B(p), None) or L.b2c_ncp_sweeps(B(sc), B(st), B(p), 4, None)
    return rc or (L.b2c_ncp_adjoint(B(sc), B(st), B(p), 4, q, q, q, q, q, None) if dtype == 8 else 0)


def _admm(lib, L, nc):
    a = _filled(lib.Admm, n_env=64, nc=nc, nv=32)
    return L.b2c_admm_solve(ctypes.byref(a), ctypes.byref(_filled(lib.AdmmParams, flags=lib.ADMM_FORWARD)), None)


def _bncp(lib, L, nc):
    p, q = _filled(lib.Bncp, n_env=64, n_max=3 * nc), ctypes.addressof(_room)
    B = ctypes.byref
    return L.b2c_bncp_solve(B(p), 10, 1e-6, 1, None) or L.b2c_bncp_vjp(B(p), q, q, q, None)


CALLS = {f"solve {f} {n} {k}": (lambda lib, L, k=k, f=f, n=n: _solve(lib, L, k, f, n))
         for f in (0, FIXED, FIXED | ROW | FIRST, FIXED | ROW | ISLANDS) for n in (50, N) for k in (0, 1, 148, -16, -4)}
CALLS["solve scenes"] = lambda lib, L: _solve(lib, L, lib.SOLVE_SCENES, FIXED | ROW | FIRST, N)
CALLS.update({f"ncp {d} {k}": (lambda lib, L, d=d, k=k: _ncp(lib, L, d, k)) for d in (4, 8) for k in (0, 1, 148, -16)})
CALLS.update({f"admm {c}": (lambda lib, L, c=c: _admm(lib, L, c)) for c in (1, 4, 8)})
CALLS.update({f"bncp {c}": (lambda lib, L, c=c: _bncp(lib, L, c)) for c in (1, 8, 9, 16)})


@pytest.mark.parametrize("call", sorted(CALLS))
def test_second_device_is_not_refused(host, call):
    lib, L = host
    for device in (0, 1, 0):
        L.fake_set_device(device)
        before = L.fake_launches()
        rc = CALLS[call](lib, L)
        assert rc == 0, (device, L.b2c_last_error().decode())
        assert L.fake_launches() > before

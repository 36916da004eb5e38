"""The library's host code against a stand-in for the CUDA runtime (fake_cudart.c): refused launches, limits and
allocations, a second device.  Each case runs in a process of its own, since limits and capacities are kept
for the process."""
import os
import subprocess
import sys

import pytest

from conftest import REPO

# (kernels go by a part of their mangled names)
PRELUDE = """
import ctypes as C, sys
import numpy as np
from nrltb import abi
lib = abi._bind(sys.argv[1], abi.GPU_SYMBOLS)
for f in ("fake_runs", "fake_refused"):
    getattr(lib, f).argtypes = [C.c_char_p, C.c_int]
for f in ("fake_refuse_launch", "fake_refuse_limit", "fake_refuse_cluster"):
    getattr(lib, f).argtypes = [C.c_char_p]
lib.fake_capacity.argtypes = [C.c_size_t]
lib.fake_largest_alloc.restype = lib.fake_used.restype = C.c_size_t

def context(device=0):
    h = C.c_void_p()
    assert lib.nrltb_ctx_create(C.byref(h), device) == 0
    return h

def diag(h, n, nk, vectors, precision=abi.PREC_FP64):
    H = np.tile(np.eye(n, dtype=complex), (nk, 1, 1))
    e, z = np.zeros((nk, n)), np.zeros((nk, n, n), complex)
    p = lambda a: a.ctypes.data_as(abi._dp)
    return lib.nrltb_diag(h, n, nk, p(H), p(H), precision, p(e), p(z) if vectors else None, None)
"""


@pytest.fixture(scope="session")
def fake_lib(tmp_path_factory):
    """The library's objects linked against the stand-in."""
    from nrltb import build
    build.build_all()
    cuda = os.path.dirname(os.path.dirname(build._nvcc()))
    out = tmp_path_factory.mktemp("fake")
    subprocess.run(["gcc", "-O1", "-fPIC", "-Wall", "-I", os.path.join(cuda, "include"), "-c",
                    os.path.join(REPO, "tests", "fake_cudart.c"), "-o", str(out / "fake.o")], check=True)
    objs = [os.path.join(build.OBJ, f[:-3] + ".o") for f in build.CU_SOURCES]
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", str(out / "lib.so"), str(out / "fake.o")] + objs +
                   ["-lpthread", "-ldl"], check=True)
    return str(out / "lib.so")


def _run(lib, code):
    env = dict(os.environ, PYTHONPATH=os.path.join(REPO, "tight-binding_gb300"))
    r = subprocess.run([sys.executable, "-c", PRELUDE + code, lib], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("n", [160, 300])
@pytest.mark.parametrize("kernel", ["k_to_unit", "k_potrf_diag64", "k_z_gemm"])
@pytest.mark.parametrize("clusters", [1000, 3])
def test_refused_launch_before_the_clusters_is_reported(fake_lib, n, kernel, clusters):
    """FP64 eigenvalues alone: a launch refused in the reduction is an error of the call, whether or not the choice of
    a cluster size, which follows it, finds room for the batch (1000 clusters, 3)."""
    _run(fake_lib, f"""
h = context()
lib.fake_clusters({clusters})
lib.fake_refuse_launch(b"{kernel}")
assert diag(h, {n}, 20, False) == abi.NRLTB_E_CUDA
assert lib.fake_refused(b"{kernel}", 0) > 0
lib.fake_refuse_launch(b"")
assert diag(h, {n}, 20, False) == 0
""")


@pytest.mark.parametrize("how", ["fake_refuse_limit", "fake_refuse_cluster", "fake_refuse_launch"])
def test_refused_clusters_leave_the_columns(fake_lib, how):
    """Where no cluster can be had the columns take over, and the refusals are no error of the call."""
    _run(fake_lib, f"""
h = context()
lib.{how}(b"13k_tri_cluster")
assert diag(h, 160, 20, True) == 0
assert lib.fake_runs(b"13k_tri_cluster", 0) == (1 if {how!r} == "fake_refuse_cluster" else 0)
assert lib.fake_runs(b"k_tri_mv", 0) == (0 if {how!r} == "fake_refuse_cluster" else 159)
""")


@pytest.mark.parametrize("kernel", ["k_convert_h", "12k_potrf_diag"])
@pytest.mark.parametrize("clusters", [1000, 3, 0])
def test_refused_launch_before_the_panels_is_reported(fake_lib, kernel, clusters):
    """The same for the mixed form, whose first panel asks the device for its cluster capacities."""
    _run(fake_lib, f"""
h = context()
lib.fake_clusters({clusters})
lib.fake_refuse_launch(b"{kernel}")
assert diag(h, 160, 20, True, abi.PREC_MIXED) == abi.NRLTB_E_CUDA
assert lib.fake_refused(b"{kernel}", 0) > 0
""")


@pytest.mark.parametrize("how", ["fake_refuse_limit", "fake_refuse_cluster", "fake_refuse_launch"])
def test_refused_panels_leave_the_columns(fake_lib, how):
    _run(fake_lib, f"""
h = context()
lib.{how}(b"11k_tri_panel")
assert diag(h, 160, 20, True, abi.PREC_MIXED) == 0
assert lib.fake_runs(b"11k_tri_panel", 0) == 0 and lib.fake_runs(b"8k_tri_mv", 0) == 159
""")


@pytest.mark.parametrize("n", [20, 160])
def test_fp64_products_on_a_second_device(fake_lib, n):
    """A kernel's shared-memory limit belongs to one device: contexts on two devices of a process launch alike."""
    _run(fake_lib, f"""
runs = []
for dev in (0, 1):
    h = context(dev)
    assert diag(h, {n}, 3, True) == 0
    runs.append([lib.fake_runs(b"8k_z_gemm", dev), lib.fake_runs(b"k_", dev)])
    assert runs[-1][0] > 0 and lib.fake_refused(b"k_", dev) == 0
assert runs[0] == runs[1]
""")


def test_fp64_products_without_their_limit_take_the_fma_pipe(fake_lib):
    _run(fake_lib, """
h = context()
lib.fake_refuse_limit(b"8k_z_gemm")
assert diag(h, 160, 3, True) == 0
assert lib.fake_runs(b"8k_z_gemm", 0) == 0 and lib.fake_runs(b"zgemm_kernel", 0) > 0
""")


def test_mixed_form_on_a_second_device(fake_lib):
    _run(fake_lib, """
runs = []
for dev in (0, 1):
    h = context(dev)
    assert diag(h, 160, 3, True, abi.PREC_MIXED) == 0
    runs.append([lib.fake_runs(k, dev) for k in (b"k_oz_gemm", b"zgemm_umma_kernel", b"k_ref_band", b"k_")])
    assert min(runs[-1]) > 0 and lib.fake_refused(b"k_", dev) + lib.fake_refused(b"zgemm", dev) == 0
assert runs[0] == runs[1]
""")


@pytest.mark.parametrize("n,digits", [(9, False), (15, False), (16, True)])
def test_digit_scratch_goes_to_orders_that_can_use_it(fake_lib, n, digits):
    """No product of an order below 16 is a digit product; their scratch for 600 matrices would be 138 MB, everything
    else a solve of these orders needs less than 16 MB a buffer."""
    _run(fake_lib, f"""
h = context()
assert diag(h, {n}, 600, True) == 0
assert (lib.fake_runs(b"8k_z_gemm", 0) > 0) == {digits}
assert (lib.fake_largest_alloc() > 100e6) == {digits}
""")


@pytest.mark.parametrize("room,digits", [(1.0, True), (0.7, True), (0.21, True), (0.1, False)])
def test_digit_scratch_that_does_not_fit(fake_lib, room, digits):
    """5 matrices of order 288 on a device that has room for a part of their 41.4 MB of digits, which are asked for
    last: the products go in parts, and on the FMA pipe where not even one matrix's digits fit."""
    _run(fake_lib, f"""
h = context()
assert diag(h, 288, 5, True) == 0
used, whole = lib.fake_used(), lib.fake_runs(b"8k_z_gemm", 0)
assert lib.nrltb_ctx_destroy(h) == 0 and lib.fake_used() == 0
lib.fake_capacity(used - int({1 - room} * 41.4e6))
h = context()
assert diag(h, 288, 5, True) == 0 and diag(h, 288, 5, False) == 0
runs = lib.fake_runs(b"8k_z_gemm", 0) - whole
assert runs > whole if {digits} else runs == 0
""")


@pytest.mark.parametrize("precision,mode,gigabytes", [("PREC_FP64", 4, 6), ("PREC_FP64", 4, 96), ("PREC_FP64", 6, 96),
                                                      ("PREC_MIXED", 6, 6), ("PREC_MIXED", 6, 40), ("PREC_MIXED", 4, 6)])
def test_chunks_of_k_fill_half_of_the_memory(fake_lib, precision, mode, gigabytes):
    """The chunk is chosen for half of the free memory: with the digits of the FP64 products, which a large chunk
    has 6 GB of, it comes to that (less what modes without derivatives don't use), the pair tables and results of
    all k points aside (3 per cent, and 8 N^2 bytes a k point of charges)."""
    _run(fake_lib, f"""
from nrltb import Context, KMesh, Opts, synth
abi._cache[abi.GPU_LIB] = lib
lib.fake_capacity({gigabytes} << 30)
st, par, _, _ = synth.bcc32()
nk = 6000
km = KMesh(np.zeros((nk, 3)), np.full(nk, 1.0 / nk))
ctx = Context(0)
ctx.bande(st, par, km, Opts(mode={mode}, precision=abi.{precision}))
share = (lib.fake_used() - (8 * 288 * 288 * nk if {mode} == 6 else 0)) / ({gigabytes} << 29)
assert lib.fake_runs(b"k_bloch_build", 0) > 2 and {0.95 if mode == 4 else 0.7} < share < 1.03, share
""")

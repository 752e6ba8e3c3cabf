"""Host code of the library without a GPU: its objects linked against a CUDA
runtime that carries out copies, only looks at kernels and can be told to fail
(fake_cudart.c)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "md.error_b200", "csrc")
NO_FAILURE = -1


@pytest.fixture(scope="module")
def rt(tmp_path_factory):
    """the library on the fake runtime"""
    if not shutil.which("nvcc") or not shutil.which("g++"):
        pytest.skip("no compiler for the objects of the library")
    from mdforce._lib import _SIGS
    subprocess.check_call(["make", "-s", "-j8", "-C", CSRC], stdout=subprocess.DEVNULL)
    d = tmp_path_factory.mktemp("fake")
    inc = os.path.join(os.path.dirname(os.path.dirname(shutil.which("nvcc"))), "include")
    subprocess.check_call(["gcc", "-O1", "-fPIC", "-I" + inc, "-c", os.path.join(HERE, "fake_cudart.c"), "-o", d / "rt.o"])
    objs = sorted(os.path.join(CSRC, "_build", f) for f in os.listdir(os.path.join(CSRC, "_build")) if f.endswith(".o"))
    subprocess.check_call(["g++", "-shared", "-Wl,-Bsymbolic", "-o", d / "libfake.so", *objs, d / "rt.o", "-lpthread"])
    lib = C.CDLL(str(d / "libfake.so"))
    for name, (res, args) in _SIGS.items():
        getattr(lib, name).restype, getattr(lib, name).argtypes = res, args
    for name, res in (("fake_calls", C.c_long), ("fake_live", C.c_long), ("fake_pinned", C.c_long),
                      ("fake_pageable_dtoh", C.c_long), ("fake_launch_name", C.c_char_p), ("fake_lowered", C.c_char_p),
                      ("fake_unprepared", C.c_char_p)):
        getattr(lib, name).restype = res
    lib.fake_fail_at.argtypes = [C.c_long]
    return lib


@pytest.fixture
def lib(rt):
    rt.fake_reset()
    assert rt.fake_live() == 0
    yield rt
    rt.fake_reset()
    assert rt.fake_live() == 0


def dbl(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def vec(t, *v):
    return (t * len(v))(*v)


def new_system(lib, n=64, device=0, box=8.0):
    pos, h = np.zeros((n, 3)), C.c_void_p()
    q = np.ones(n)
    assert lib.md_system_create(C.byref(h), n, vec(C.c_double, box, box, box), dbl(pos), None, None, dbl(q), None, 1,
                                device) == 0, lib.md_last_error_message()
    return h


def make_map(lib, K, kind="ik"):
    h = C.c_void_p()
    KK, LL = vec(C.c_int, *K), vec(C.c_double, 8.0, 8.0, 8.0)
    if kind == "ik":
        rc = lib.md_errmap_create(C.byref(h), KK, LL, 1.0, 6, 0)
    elif kind == "ana":
        rc = lib.md_errmap_create_ana(C.byref(h), KK, LL, 1.0, 6, 0)
    else:
        rc = lib.md_errmap_create_dir(C.byref(h), KK, LL, 1.0, 3.0, 0)
    return rc, h


@pytest.mark.parametrize("kind", ["ik", "ana", "dir"])
def test_error_is_reported_once(lib, kind):
    """after a map that memory does not hold, the next one is made"""
    lib.fake_fail_at(1)  # the arrays' allocation (0: the stream)
    assert make_map(lib, (16, 16, 16), kind)[0] != 0
    assert b"out of memory" in lib.md_last_error_message()
    lib.fake_fail_at(NO_FAILURE)
    rc, h = make_map(lib, (8, 8, 8), kind)
    assert rc == 0, lib.md_last_error_message()
    lib.md_errmap_destroy(h)


def with_each_call_failing(lib, op):
    """op() once as it is, then once for each of its CUDA calls with that call failing"""
    lib.fake_fail_at(NO_FAILURE)
    op()
    n = lib.fake_calls()
    for k in range(n):
        lib.fake_fail_at(k)
        op()
        lib.fake_fail_at(NO_FAILURE)
        yield k


@pytest.mark.parametrize("kind", ["ik", "ana", "dir"])
@pytest.mark.parametrize("K", [(8, 8, 8), (8, 9, 12)])
def test_failed_map_leaves_nothing(lib, kind, K):
    """no memory, stream or pool reference stays after a map's creation fails at any of its calls"""
    def op():
        rc, h = make_map(lib, K, kind)
        if rc == 0:
            lib.md_errmap_destroy(h)

    for k in with_each_call_failing(lib, op):
        assert lib.fake_live() == 0, k
    trims = lib.fake_trims()
    op()
    assert lib.fake_trims() == trims + 1  # the last user of the pool leaves: none of the failures kept a reference


BIG = 3 << 20  # atoms whose positions take more than the scratch a system keeps (64 MB)


@pytest.mark.parametrize("call", ["positions", "set_positions", "charges", "rcut", "ewald"])
def test_failed_call_leaves_no_scratch(lib, call):
    """workspace taken for one call is freed when any later call in it fails"""
    n = {"charges": 9 << 20, "rcut": 17 << 20, "ewald": 64}.get(call, BIG)
    h = new_system(lib, n)
    buf = np.zeros(3 * n)
    f32 = np.zeros(n, np.float32)
    e = C.c_double()
    K = vec(C.c_int, 2, 1024, 2048)

    def op():
        if call == "positions":
            lib.md_system_get_positions(h, dbl(buf))
        elif call == "set_positions":
            lib.md_system_set_positions(h, dbl(buf))
        elif call == "charges":
            lib.md_system_get_charges(h, dbl(buf))
        elif call == "rcut":
            lib.md_system_get_rcut(h, f32.ctypes.data_as(C.POINTER(C.c_float)))
        else:
            lib.md_ewald_exact(h, K, 1.0, C.byref(e), 1)

    op()
    held = lib.fake_live()
    for k in with_each_call_failing(lib, op):
        assert lib.fake_live() == held, k
    lib.md_system_destroy(h)


def hermite(lib, nbin, CC=4.0, n=8):
    h = C.c_void_p()
    assert lib.md_hspme_create(C.byref(h), n, vec(C.c_int, 12, 12, 12), vec(C.c_double, 8.0, 8.0, 8.0), 1.0, CC, nbin,
                               0, 0) == 0
    return h


@pytest.mark.parametrize("CC", [1.0, 4.0, 5.0])
def test_hermite_handles_keep_their_shared_memory(lib, CC):
    """handles of one stencil width and different coefficient counts, used in turn: neither takes
    the kernels' shared-memory limit below what the other one launches with"""
    big, small = hermite(lib, 64, CC), hermite(lib, 40, CC)
    buf = np.zeros(4096)
    p = buf.ctypes.data
    for h in (big, small, big):
        assert lib.md_hspme_energy(h, p, p, p, 1, p, p, p, p, p, None) == 0
        assert lib.md_hspme_force_error(h, p, p, p, 1, p, p, p, p, p, None) == 0
        assert lib.fake_lowered() is None
    lib.md_hspme_destroy(big)
    lib.md_hspme_destroy(small)


def functional(lib, k):
    h = C.c_void_p()
    assert lib.md_ikerr_create(C.byref(h), vec(C.c_int, k, k, k), vec(C.c_double, 30.0, 30.0, 30.0), 0.95, 2.0, 4, 10,
                               0, 100, 100.0, 100.0, 0) == 0, lib.md_last_error_message()
    return h


def test_functionals_keep_their_shared_memory(lib):
    """a functional of a smaller mesh made later does not take the limit that a larger one launches with"""
    big = functional(lib, 256)
    c, v, g = np.zeros(8), np.zeros(1), np.zeros(8)
    assert lib.md_ikerr_evaluate(big, 1, dbl(c), dbl(v), dbl(g)) == 0
    small = functional(lib, 224)
    assert lib.fake_lowered() is None
    for h in (small, big):
        assert lib.md_ikerr_evaluate(h, 1, dbl(c), dbl(v), dbl(g)) == 0, lib.md_last_error_message()
    lib.md_ikerr_destroy(big)
    lib.md_ikerr_destroy(small)


@pytest.mark.parametrize("K", [(16, 16, 32), (32, 16, 16)])
@pytest.mark.parametrize("device_outputs", [False, True])
def test_energy_alone_is_not_transformed_back(lib, K, device_outputs):
    """an SPME energy without gradients ends with the k-space step, on meshes that run by planes too"""
    s, sp = new_system(lib), C.c_void_p()
    assert lib.md_spme_create(C.byref(sp), s, vec(C.c_int, *K), 4, 1.0, 0) == 0
    out, grad = np.zeros(2), np.zeros(3 * 64)

    def launched(gradient):
        n = lib.fake_launches()
        if device_outputs:
            assert lib.md_spme_energy_grad_device(sp, s, out.ctypes.data, None, grad.ctypes.data if gradient else None,
                                                  None) == 0
        else:
            assert lib.md_spme_energy_grad(sp, s, dbl(out), None, dbl(grad) if gradient else None, dbl(out[1:]), None) == 0
        return [lib.fake_launch_name(k).decode() for k in range(n, lib.fake_launches())]

    def back(names):
        return [x for x in names if "gather" in x or "z_backward" in x or ("fftp" in x and "Li2E" in x)]

    assert not back(launched(False))
    with_gradient = launched(True)
    assert any("gather" in x for x in with_gradient) and len(back(with_gradient)) >= 2
    lib.md_spme_destroy(sp)
    lib.md_system_destroy(s)


@pytest.mark.parametrize("precision", [0, 1])
def test_list_kernels_are_prepared_on_each_device(lib, precision):
    """the list build's shared-memory limit is set on every device that has a list, not on the first one only"""
    for device in (0, 1):
        s, cl, nl = new_system(lib, 64, device), C.c_void_p(), C.c_void_p()
        assert lib.md_cell_list_create(C.byref(cl), s, 2.0, 7, 1) == 0, lib.md_last_error_message()
        for mode in (0, 1):
            assert lib.md_nlist_create(C.byref(nl), s, 1.5, 0.3, 4.0, mode) == 0, lib.md_last_error_message()
            assert lib.md_cell_list_rebuild(cl, s) == 0, lib.md_last_error_message()
            assert lib.md_nlist_rebuild(nl, s, cl) == 0, lib.md_last_error_message()
            lib.md_nlist_destroy(nl)
        lib.md_cell_list_destroy(cl)
        lib.md_system_destroy(s)
    assert lib.fake_unprepared() is None


@pytest.mark.parametrize("n", [1000, BIG, 3 * BIG])
def test_frames_of_any_size_through_page_locked_memory(lib, n):
    """frames arrive whole through a page-locked buffer of bounded size, also above what a system keeps"""
    h = new_system(lib, n)
    out = np.ones((n, 3))
    before, held = lib.fake_pageable_dtoh(), lib.fake_pinned()
    assert lib.md_system_get_positions(h, dbl(out)) == 0
    assert lib.fake_pageable_dtoh() == before
    assert lib.fake_pinned() - held <= 4 << 20
    assert not out.any()
    lib.md_system_destroy(h)


def test_several_arrays_in_pieces(lib):
    """arrays of no whole number of pieces, and empty ones, keep their bytes"""
    s, a = new_system(lib, 64, 0, 120.0), C.c_void_p()
    assert lib.md_arc_create(C.byref(a), s, 1.0, 2.5, 5.0, 0.5) == 0, lib.md_last_error_message()
    dims = np.zeros(3, np.int32)
    assert lib.md_arc_get_dims(a, dims.ctypes.data_as(C.POINTER(C.c_int)), None) == 0
    n = int(dims.prod())
    assert 8 * n > 4 * (512 << 10) and 8 * n % (512 << 10)
    rc, idx, err = np.ones(n), np.ones(n, np.int32), np.ones(n)
    before = lib.fake_pageable_dtoh()
    assert lib.md_arc_get_rcut(a, dbl(rc), idx.ctypes.data_as(C.POINTER(C.c_int)), dbl(err)) == 0
    assert lib.fake_pageable_dtoh() - before < 1 << 16  # the state alone
    assert not rc.any() and not idx.any() and not err.any()
    rc[:] = 1
    assert lib.md_arc_get_rcut(a, None, None, dbl(rc)) == 0 and not rc.any()
    assert lib.md_arc_get_rcut(a, None, None, None) == 0
    lib.md_arc_destroy(a)
    lib.md_system_destroy(s)


@pytest.mark.parametrize("given,passed", [(None, None), (0, 1), (0x7f00deadbeef, 0x7f00deadbeef)])
def test_functional_on_the_default_stream(monkeypatch, given, passed):
    """torch's default stream has the handle 0, which the C ABI reads as the functional's own stream:
    its work would not be in order with torch's"""
    import mdforce.optibasis as ob
    seen = []

    def fake(h, nc, coeffs, values, grads, stream):
        seen.append(stream.value)
        return 0

    monkeypatch.setattr(ob.lib, "md_ikerr_evaluate_device", fake)

    class Dummy:
        h = C.c_void_p(1234)

    ob.IkErrorGPU.evaluate_device(Dummy(), 16, 16, None, 1, given)
    assert seen == [passed]


def test_uploads_are_in_order_with_the_kernels(lib):
    """no copy or fill goes around the streams that the kernels run on: what a plain cudaMemcpy has
    not delivered when it returns, a kernel on a non-blocking stream does not wait for"""
    before = lib.fake_unordered()
    s, cl, nl, sp, eng = new_system(lib), C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_void_p()
    assert lib.md_cell_list_create(C.byref(cl), s, 2.0, 7, 1) == 0
    assert lib.md_nlist_create(C.byref(nl), s, 1.5, 0.3, 4.0, 0) == 0
    assert lib.md_spme_create(C.byref(sp), s, vec(C.c_int, 16, 16, 16), 4, 1.0, 0) == 0
    assert lib.md_engine_create(C.byref(eng), s) == 0
    assert lib.md_engine_register_lj_pair(eng, 0, 0, 1.0, 1.0, 0.0) == 0, lib.md_last_error_message()
    assert lib.md_cell_list_rebuild(cl, s) == 0 and lib.md_nlist_rebuild(nl, s, cl) == 0
    assert lib.md_engine_apply_nonbonded(eng, s, nl, 1) == 0, lib.md_last_error_message()
    assert lib.md_spme_apply(sp, s, 1) == 0
    assert lib.fake_unordered() == before
    for destroy, h in (("spme", sp), ("nlist", nl), ("cell_list", cl), ("engine", eng), ("system", s)):
        getattr(lib, f"md_{destroy}_destroy")(h)


def test_exact_sum_over_a_long_axis(lib):
    """mode boxes of more columns than a grid has rows of blocks"""
    s, e = new_system(lib, 2), C.c_double()
    for K in ((1, 1, 2200000), (1, 2200000, 1), (2200000, 1, 1)):
        assert lib.md_ewald_exact(s, vec(C.c_int, *K), 1.0, C.byref(e), 1) == 0, lib.md_last_error_message()
    lib.md_system_destroy(s)


def test_hermite_workspace_falls_back_to_smaller_batches(lib):
    """one allocation; where memory does not hold a batch of four, two, and calls of more candidates go through"""
    h = hermite(lib, 8)
    full, calls = lib.fake_live(), lib.fake_calls()
    lib.md_hspme_destroy(h)
    lib.fake_fail_at(calls - 1)  # the last call of the creation: the workspace
    h = hermite(lib, 8)
    lib.fake_fail_at(NO_FAILURE)
    assert abs(lib.fake_live() - full // 2) <= full // 8
    buf = np.zeros(1 << 14)
    p = buf.ctypes.data
    assert lib.md_hspme_energy(h, p, p, p, 5, p, p, p, p, p, None) == 0
    lib.md_hspme_destroy(h)

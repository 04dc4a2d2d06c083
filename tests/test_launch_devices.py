"""Launchers called for a second device of the process, on a runtime that has several devices and no GPU."""
import ctypes as C

import pytest

import fake_cuda

ADDRESS = 1 << 30          # 16-byte aligned, never followed


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_cuda.build(str(tmp_path_factory.mktemp("fake_cuda") / "libesgd_fake.so"))


@pytest.fixture(autouse=True)
def first_device(lib):
    lib.fake_device(0)
    fake_cuda.launches(lib)
    yield
    lib.fake_device(0)


class _Outcome(C.Structure):
    _fields_ = [("round", C.c_uint64)] + [(n, C.c_uint32) for n in "role contributors is_sync applied status pad".split()]


@pytest.mark.parametrize("local", [0, 1])
@pytest.mark.parametrize("bytes_", [0, 40, 16 << 20])
@pytest.mark.parametrize("offset", [0, 2])
def test_a_collective_is_posted_and_waited_for_from_a_thread_on_another_device(lib, local, bytes_, offset):
    """A thread starts on device 0, and a rank's helper thread may wait for a result that is staged on device 3."""
    lib.esgd_collective_create.argtypes = [C.c_void_p, C.c_uint64, C.c_int, C.c_int, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_uint64,
                                           C.c_void_p, C.POINTER(C.c_void_p)]
    for f in (lib.esgd_collective_post, lib.esgd_collective_wait):
        f.argtypes = [C.c_void_p, C.c_void_p]
    lib.esgd_collective_destroy.argtypes = [C.c_void_p]
    outcome, handle = _Outcome(applied=1), C.c_void_p()
    lib.fake_device(3)
    side, callers = lib.fake_stream(3), lib.fake_stream(3) + 1
    assert lib.esgd_collective_create(ADDRESS, 4096, 148, local, side, 1, ADDRESS + offset, 2 * ADDRESS, bytes_, C.addressof(outcome),
                                      C.byref(handle)) == 0
    lib.fake_device(0)
    assert lib.esgd_collective_post(handle, callers) == 0 and lib.fake_current_device() == 0
    assert lib.esgd_collective_wait(handle, callers) == 0 and lib.fake_current_device() == 0
    lib.esgd_collective_destroy(handle)
    rows = fake_cuda.launches(lib)
    assert all(device == 3 for _, device, *_ in rows)
    copied = [r for r in rows if "hand_over" in r[0]]
    assert len(copied) == (bytes_ > 0 and offset == 0) and len(rows) - len(copied) == (1 if local else 2)

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


def _pointer_calls(lib, rows):
    """Calls whose pointers (``p``) are addresses that nobody follows, everything else as given."""
    def call(name, *args):
        f = getattr(lib, name)
        f.argtypes = [C.c_void_p if a is None or a == ADDRESS or a == "stream" else C.c_int for a in args]
        return lambda stream: f(*[C.c_void_p(stream) if a == "stream" else a for a in args])
    return [call(*r) for r in rows]


P, S = ADDRESS, "stream"
LARGE_KERNELS = {
    "gemm_kernel": [("esgd_gemm_bf16", P, P, P, 40000, 512, 256, 256, 256, 512, 0, 0, 0, None, None, 0, 1, None, None, None, 0, None, S),
                    ("esgd_gemm_bf16", P, P, P, 4096, 512, 4096, 4096, 4096, 512, 0, 0, 0, None, None, 0, 1, None, None, None, 0, None, S),
                    ("esgd_gemm_bf16", P, P, P, 256, 64, 8192, 256, 64, 64, 1, 1, 2, None, None, 0, 8, None, None, None, 0, None, S)],
    "gemm_split_kernel": [("esgd_gemm_bf16", P, P, P, 49, 512, 2048, 2048, 2048, 512, 0, 0, 0, None, None, 0, 1, None, None, None, 0, None, S)],
    "conv_kernel": [("esgd_conv2d_fwd", P, P, P, 32, 56, 56, 64, 64, 3, 3, 1, 1, None, None, None, 0, P, P, None, S),
                    ("esgd_conv2d_fwd", P, P, P, 64, 28, 28, 128, 128, 3, 3, 1, 1, None, None, None, 0, P, P, None, S),
                    ("esgd_conv2d_fwd", P, P, P, 64, 56, 56, 128, 128, 3, 3, 2, 1, None, None, None, 0, P, P, None, S),
                    ("esgd_conv2d_dgrad", P, P, P, 64, 14, 14, 256, 256, 3, 3, 1, 1, None, None, None, S)],
    "conv_split_kernel": [("esgd_conv2d_fwd", P, P, P, 1, 7, 7, 512, 512, 3, 3, 1, 1, None, None, None, 0, None, None, None, S)],
    "conv_wgrad_kernel": [("esgd_conv2d_wgrad", P, P, P, 64, 56, 56, 128, 128, 3, 3, 2, 1, None, S)],
    "conv_wgrad_halo_kernel": [("esgd_conv2d_wgrad_halo", P, P, P, 1, 56, 56, 64, 64, 3, 3, 1, None, S),
                               ("esgd_conv2d_wgrad_halo", P, P, P, 64, 28, 28, 128, 128, 3, 3, 1, None, S),
                               ("esgd_conv2d_wgrad_halo", P, P, P, 64, 7, 7, 512, 512, 3, 3, 1, None, S)],
    "conv_wgrad_packed_kernel": [("esgd_conv2d_wgrad_halo", P, P, P, 64, 56, 56, 64, 64, 3, 3, 1, None, S)],
    "stem_fwd_kernel": [("esgd_stem_fwd", P, P, P, P, 64, 224, 224, 3, 64, 7, 7, 2, 3, 192, None, None, 0, P, P, None, S)],
    "stem_wgrad_kernel": [("esgd_stem_wgrad", P, P, P, 64, 224, 224, 3, 64, 7, 7, 2, 3, 192, None, S)],
    "conv_narrow_kernel": [("esgd_conv_narrow_fwd", P, P, P, 128, 32, 32, 16, 16, 1, None, None, None, 0, P, P, S)],
    "wgrad_narrow_kernel": [("esgd_conv_narrow_wgrad", P, P, P, 128, 32, 32, 16, 16, 1, S)],
}


@pytest.mark.parametrize("kernel", sorted(LARGE_KERNELS))
def test_kernels_with_much_shared_memory_run_on_every_device_of_the_process(lib, kernel):
    """A kernel may have more than 48 KB once that has been asked for, on each device by itself."""
    calls = _pointer_calls(lib, LARGE_KERNELS[kernel])
    for device in (0, 3, 0, 70):
        lib.fake_device(device)
        for call in calls:
            assert call(lib.fake_stream(device)) == 0, device
        rows = fake_cuda.launches(lib)
        assert len(rows) == len(calls)
        for name, ran_on, _, smem, *_ in rows:
            assert kernel in name and ran_on == device and smem > 48 * 1024, (name, ran_on, smem)


def test_shared_memory_is_asked_for_once_for_a_kernel_and_device(lib):
    (call,) = _pointer_calls(lib, LARGE_KERNELS["stem_wgrad_kernel"])
    lib.fake_device(5)
    assert call(lib.fake_stream(5)) == 0
    asked = lib.fake_attributes()
    assert call(lib.fake_stream(5)) == 0 and lib.fake_attributes() == asked

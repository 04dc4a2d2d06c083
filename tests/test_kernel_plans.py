"""Launch geometry of the convolution kernels, swept on the CPU.

The planners are the host arithmetic the launchers themselves use (box sizes, stages, tap sets, pixel splits);
they need no device.  The sweep checks every invariant the kernels rely on: boxes and the rows their most shifted
views reach stay inside their shared-memory slots, stages fit the CTA's shared memory, accumulators fit tensor
memory, TMA boxes respect the 256-per-dimension limit, tiles and splits cover the problem exactly.  Split reductions
and the stem are swept through their launchers, on a runtime without a GPU that knows the limits of a launch.
"""
import ctypes as C
import itertools

import pytest

import fake_cuda
from eagersgd_b200.parallel import _native as N

HALO_BYTES = 32 * 1024


def _lib():
    lib = N.cuda()
    lib.esgd_conv2d_halo_plan.argtypes = [C.c_int] * 9 + [C.c_void_p]
    lib.esgd_conv2d_halo_plan.restype = None
    lib.esgd_conv2d_wgrad_halo_plan.argtypes = [C.c_int] * 9 + [C.c_void_p]
    lib.esgd_conv2d_wgrad_halo_plan.restype = None
    return lib


SHAPES = [(n, hw, cin, cout, k) for n, hw, cin, cout, k in itertools.product(
    (1, 7, 256), (7, 8, 14, 24, 28, 56, 112, 126, 130, 224), (64, 128, 256, 512), (64, 72, 128, 256, 512), (2, 3, 5, 7))]


def test_forward_halo_plans_fit_their_slots():
    lib = _lib()
    out = (C.c_int * 11)()
    seen = 0
    for n, hw, cin, cout, k in SHAPES:
        pad = (k - 1) // 2
        lib.esgd_conv2d_halo_plan(n, hw, hw, cin, cout, k, k, 1, pad, out)
        ok, bh, pw, bn, res_kb, nhalo, nst, box, view, used, area = list(out)
        if not ok:
            continue
        seen += 1
        ho, wo = hw + 2 * pad - k + 1, hw + 2 * pad - k + 1
        assert pw == wo + k - 1 and pw <= 128 and ho % bh == 0 and bh * pw <= 128
        assert bh * wo >= 64                                  # enough real rows per 128-row tile
        assert box <= HALO_BYTES and view <= HALO_BYTES       # the box and the farthest view stay in the slot
        assert pw <= 256 and bh + k - 1 <= 256                # TMA box extents
        assert 0 < used <= area and nhalo in (2, 3) and nst >= 1
        assert bn in (64, 128) and cout <= 128
        if res_kb:
            assert res_kb == k * k * (cin // 64) and nhalo == 2
        else:
            assert nst >= 2
    assert seen > 50
    # stride 2 and wide outputs never take this path
    lib.esgd_conv2d_halo_plan(4, 56, 56, 64, 64, 3, 3, 2, 1, out)
    assert out[0] == 0
    lib.esgd_conv2d_halo_plan(4, 14, 14, 256, 256, 3, 3, 1, 1, out)
    assert out[0] == 0


def test_forward_halo_plans_have_the_tile_width_of_the_launch():
    """Small problems are launched with narrower tiles while twice as many still fit one wave of the SMs."""
    lib = _lib()
    out = (C.c_int * 11)()
    widths = set()
    for n, hw, cin, cout, k in SHAPES:
        pad = (k - 1) // 2
        lib.esgd_conv2d_halo_plan(n, hw, hw, cin, cout, k, k, 1, pad, out)
        if not out[0]:
            continue
        ho = hw + 2 * pad - k + 1
        m_tiles, bn = -(-n * ho * ho // 128), 64 if cout <= 64 else 128
        if bn == 128 and 2 * m_tiles * -(-cout // 128) <= lib.esgd_sm_count():
            bn = 64
        assert out[3] == bn, (n, hw, cin, cout, k)
        widths.add((cout, bn))
    assert {(72, 64), (72, 128), (128, 64), (128, 128), (64, 64)} <= widths


@pytest.mark.parametrize("sms", [148, 132])
def test_weight_gradient_plans_cover_the_problem(sms):
    lib = _lib()
    out = (C.c_int * 18)()
    seen, packed_seen = 0, 0
    for n, hw, cin, cout, k in SHAPES:
        pad = (k - 1) // 2
        lib.esgd_conv2d_wgrad_halo_plan(n, hw, hw, cin, cout, k, k, pad, sms, out)
        ok, bh, pw, ksteps, abox, xbox, nst, sets, tps, splits, bps, grid, bn, smem, mt, nt, packed, bank = list(out)
        if not ok:
            continue
        seen += 1
        ho = wo = hw + 2 * pad - k + 1
        assert ho % bh == 0 and bh * pw <= 128 and ksteps <= 8 and ksteps * 16 >= bh * pw
        assert abox % 1024 == 0 and xbox % 1024 == 0
        assert abox >= ksteps * 16 * 128 >= bh * pw * 128                       # dy box + zero K padding
        off_max = (k - 1) * pw + (k - 1)
        assert xbox >= (ksteps * 16 + off_max) * 128 >= (bh + k - 1) * pw * 128  # x box and the farthest view
        stages = nst * (abox + xbox if packed else 2 * abox + (bn // 64) * xbox)
        # stages, then the sums in their place, and the barriers behind the larger of the two
        assert 2 <= nst <= 4 and 1024 + max(stages, bank) + 256 <= smem <= 227 * 1024
        if packed:
            packed_seen += 1
            assert k == 3 and cin == 64 and cout <= 64 and (sets, tps, mt, nt) == (1, 9, 1, 1)
            # a kilobyte in front of dy, whose last row of zeros is the pixel before the first, and a pixel behind the last K step
            assert abox >= 1024 + (ksteps * 16 + 1) * 128
            # three blocks of columns a box row apart, the second product two pixels further on
            assert xbox >= (ksteps * 16 + 2 * pw + 2) * 128
            assert bank >= cout * 9 * 64 * 4 and (bank // 64) % 32 == 16                     # an odd number of 16 bytes a row
        else:
            assert tps * bn <= 512 and sets * tps >= k * k and (sets - 1) * tps < k * k   # accumulators fit TMEM, taps covered
            assert bank == 128 * (4 * bn + 16)
        boxes = (ho // bh) * n
        assert splits * bps >= boxes and (splits - 1) * bps < boxes               # no empty split, all boxes covered
        assert grid == sets * mt * nt * splits <= max(sms, sets * mt * nt) and mt == -(-cout // 128) and nt == -(-cin // bn)
        assert pw <= 256 and bh + k - 1 <= 256
    assert seen > 100 and packed_seen > 5


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_cuda.build(str(tmp_path_factory.mktemp("fake_cuda") / "libesgd_fake.so"))


P = 1 << 30                # an address that nobody follows


def _call(lib, name, *args):
    f = getattr(lib, name)
    f.argtypes = [C.c_void_p if a is None or a == P else C.c_int for a in args] + [C.c_void_p]
    lib.fake_device(0)
    rc = f(*args, lib.fake_stream(0))
    return rc, fake_cuda.launches(lib)


def test_split_reductions_are_launches_that_a_device_can_take(fake):
    """Clusters of 2, 4 or 8 CTAs that can all be resident at once, one for each tile of 64 columns; and only these."""
    seen = set()
    for n, hw, cin, cout, k in itertools.product((1, 2, 5, 16, 33), (1, 4, 7, 8, 14, 28, 130), (64, 72, 512, 2048), (8, 64, 72, 256, 512, 1000), (1, 3)):
        if k == 3:
            rc, rows = _call(fake, "esgd_conv2d_fwd", P, P, P, n, hw, hw, cin, cout, 3, 3, 1, 1, P, P, P, 1, None, None, None)
            across = min(hw, 128)
            down = max(d for d in range(1, 128 // across + 1) if hw % d == 0)
            images = max(1, min(n, 128 // (across * down))) if down == hw else 1
            tiles = -(-hw // across) * (hw // down) * -(-n // images) * -(-cout // 64)
        else:
            rc, rows = _call(fake, "esgd_gemm_bf16", P, P, P, n * hw * hw, cout, cin, cin, cin, cout, 0, 0, 0, P, P, 1, 1, None, None, P, cout, None)
            tiles = -(-(n * hw * hw) // 128) * -(-cout // 64)
        assert rc == 0 and len(rows) == 1, (n, hw, cin, cout, k, rc)
        name, _, threads, smem, cluster, blocks = rows[0]
        if "split" not in name:
            continue
        blocks_k = k * k * -(-cin // 64)
        assert blocks == tiles * cluster and cluster in (2, 4, 8) and blocks <= 148 and threads == 192, (n, hw, cin, cout, k)
        assert blocks_k >= 16 and (cluster < 8 or blocks <= 15 * 8), (n, hw, cin, cout, k)      # 15 clusters of eight are resident at once
        seen.add((k, cluster))
    assert seen == set(itertools.product((1, 3), (2, 4, 8)))


def test_stems_are_launches_that_a_device_can_take(fake):
    """Every image that the forward pass accepts, the weight gradient accepts, too: it is left nothing else to work from."""
    seen = 0
    for n, h, w in itertools.product((1, 3, 48, 64, 256), (8, 16, 24, 112, 128, 224, 320), (8, 12, 64, 112, 224, 320, 328, 400)):
        rc, rows = _call(fake, "esgd_stem_fwd", P, P, P, P, n, h, w, 3, 64, 7, 7, 2, 3, 192, None, None, 0, P, P, None)
        back, more = _call(fake, "esgd_stem_wgrad", P, P, P, n, h, w, 3, 64, 7, 7, 2, 3, 192, None)
        assert rc == back and rc in (0, -100), (n, h, w, rc, back)
        if rc == 0:
            seen += 1
            assert h % 16 == 0 and w % 8 == 0 and len(rows) == len(more) == 1
            assert all(1 <= r[5] <= 148 and r[3] <= 227 * 1024 for r in rows + more)
    assert seen > 50


@pytest.mark.parametrize("n,h,w,training,inference", [(1, 8, 8, True, True), (148, 1, 32, True, True), (149, 1, 32, False, False), (149, 1, 27, False, True), (4, 37, 32, True, True),
                                                      (1, 8, 33, False, True), (64, 8, 8, False, True), (65, 8, 8, False, False), (1, 64, 64, False, True),
                                                      (1, 8, 65, False, False)])
def test_rows_in_shared_memory_for_64_channels(fake, n, h, w, training, inference):
    """One output row a block, of at most 32 pixels; in inference up to 4096 pixels in rows of at most 64 as well."""
    sizes = (n, h, w, 64, 64)
    inference = inference or training
    for want, call in ((training, ("esgd_conv_narrow_fwd", P, P, P) + sizes + (1, None, None, None, 0, P, P)),
                       (training, ("esgd_conv_narrow_dgrad", P, P, P) + sizes + (None, None)),
                       (inference, ("esgd_conv_narrow_fwd", P, P, P) + sizes + (1, P, P, P, 1, None, None))):
        rc, rows = _call(fake, *call)
        assert rc == (0 if want else -100) and len(rows) == int(want), call
        if want:
            assert rows[0][5] == min(n * h, 148)

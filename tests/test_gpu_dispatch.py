"""Both sides of the launch rules that depend on sizes, against the CPU oracle bit for bit."""
import numpy as np
import pytest

import _libs
import astc_implementation_b200 as ab
from astc_implementation_b200 import synth

pytestmark = pytest.mark.gpu


def oracle_encode(img, bx, by, fixed):
    h, w = img.shape[:2]
    n = ((w + bx - 1) // bx) * ((h + by - 1) // by)
    out = np.zeros((n, 16), np.uint8)
    sym = np.zeros((n, 108), np.uint32)
    orc = _libs.oracle()
    prev = orc.orc_set_semantics(1 if fixed else 0)
    try:
        assert orc.orc_encode(_libs.ptr(np.ascontiguousarray(img)), w, h, bx, by, 0, _libs.ptr(out), _libs.ptr(sym)) == 0
    finally:
        orc.orc_set_semantics(prev)
    return out, sym


def check_full_search(img, bx, by, fixed):
    h, w = img.shape[:2]
    enc = ab.ASTCEncoder(device=0, fixed=fixed)
    enc.secondaryInit(w, h, bx, by)
    sym = enc.encode_symbolic(img)
    out = enc.encode(img).reshape(-1, 16)
    enc.close()
    ref_out, ref_sym = oracle_encode(img, bx, by, fixed)
    assert np.array_equal(sym, ref_sym)
    assert np.array_equal(out, ref_out)


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("w,h,bx,by", [(4 * 29, 4 * 17, 4, 4),    # 493 blocks, 1,479 partition searches: a CTA each
                                       (4 * 26, 4 * 19 - 1, 4, 4),  # 494 blocks, 1,482: a warp each
                                       (8 * 26 - 3, 8 * 19, 8, 8)])
def test_partition_search_around_the_wide_limit(w, h, bx, by, fixed):
    """Texels with zero channels in about a third of the blocks: the reference's semantics sum
    the deviations of the other texels from the partition's totals."""
    img = synth.make_texture(w, h, 31 + bx)
    rng = np.random.default_rng(w)
    hole = rng.random((h, w, 4)) < 0.02
    img[hole] = 0
    check_full_search(img, bx, by, fixed)


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("bx,by,blocks_x,blocks_y", [(4, 4, 9, 5),    # 585 partitioned blocks: 128 threads each
                                                     (4, 4, 23, 2),   # 598: 32
                                                     (5, 4, 23, 2),   # 32
                                                     (5, 5, 23, 2),   # 128
                                                     (12, 10, 23, 2),  # 256
                                                     (12, 12, 12, 4)])  # 256
def test_front_threads_by_footprint_and_launch_size(bx, by, blocks_x, blocks_y, fixed):
    img = synth.make_texture(bx * blocks_x - 1, by * blocks_y, 57 + bx)
    check_full_search(img, bx, by, fixed)

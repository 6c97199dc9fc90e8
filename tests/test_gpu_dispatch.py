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


def gpu_decode(bx, by, w, h, blocks, shift=0):
    import torch
    d_blk = torch.zeros(blocks.size + 16, dtype=torch.uint8, device="cuda")
    d_blk[shift:shift + blocks.size] = torch.from_numpy(blocks.reshape(-1)).cuda()
    d_out = torch.zeros(w * h * 4, dtype=torch.uint8, device="cuda")
    d_sse = torch.zeros(4, dtype=torch.int64, device="cuda")
    ref = torch.full((w * h * 4,), 100, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream()
    ab.decode_device(bx, by, w, h, d_blk.data_ptr() + shift, d_out.data_ptr(), s.cuda_stream)
    ab.decode_error_device(bx, by, w, h, d_blk.data_ptr() + shift, ref.data_ptr(), d_sse.data_ptr(), s.cuda_stream)
    torch.cuda.synchronize()
    return d_out.cpu().numpy().reshape(h, w, 4), d_sse.cpu().numpy()


@pytest.mark.parametrize("bx,by", [(4, 4), (6, 5), (8, 8), (12, 12)])
@pytest.mark.parametrize("blocks_x,blocks_y", [(1, 70), (3, 43), (63, 2), (64, 2), (65, 3), (130, 1)])
def test_decode_groups_of_blocks(bx, by, blocks_x, blocks_y):
    """Images narrower than a CTA's 64 blocks, exactly as wide and wider, ragged, of random bits
    (a third with a valid void-extent or common block mode), aligned and not."""
    rng = np.random.default_rng(blocks_x * 100 + blocks_y + bx)
    n = blocks_x * blocks_y
    blocks = rng.integers(0, 256, (n, 16)).astype(np.uint8)
    blocks[::3, 0] = 0x42 + 16 * rng.integers(0, 4, len(blocks[::3]))  # 4x4-grid modes and their neighbours
    blocks[::3, 1] = (blocks[::3, 1] & 0xF8) | rng.integers(0, 2, len(blocks[::3]))
    blocks[::17, :2] = (0xFC, 0xFD)  # LDR void extent
    w, h = bx * blocks_x - 1, by * blocks_y - 2
    host = ab.decode(bx, by, w, h, blocks)
    for shift in (0, 1):
        img, sse = gpu_decode(bx, by, w, h, blocks, shift)
        assert np.array_equal(img, host)
        d = host.astype(np.int64) - 100
        assert np.array_equal(sse, (d * d).reshape(-1, 4).sum(axis=0))


def _gemm(A, B, M, N, K, sa, sb, bias=None, relu=0, C=None):
    import ctypes
    import torch
    out = torch.zeros(M, N, dtype=torch.float32, device="cuda") if C is None else C.clone()
    p = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None
    ab._check(ab.load_library().astcb200_train_gemm(p(A), p(B), p(out), M, N, K, sa[0], sa[1], sb[0], sb[1], p(bias), relu,
                                                    0 if C is None else 1, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    return out.cpu().numpy().astype(np.float64)


@pytest.mark.parametrize("layout", ["nt", "nn", "tn", "odd stride", "unaligned"])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (127, 63, 17), (129, 65, 128), (64, 256, 2048), (256, 256, 2047), (700, 1408, 256)])
def test_training_gemm_tiles_splits_and_layouts(M, N, K, layout):
    """Against float64 with the bound of K + 8 roundings per sum (split sums add a few)."""
    import torch
    g = torch.Generator().manual_seed(M + N + K)
    a, b = torch.randn(M, K, generator=g), torch.randn(K, N, generator=g)
    bias, c0 = torch.randn(N, generator=g), torch.randn(M, N, generator=g)
    ref = a.double() @ b.double()
    bound = (K + 8) * 2.0 ** -24 * (a.abs().double() @ b.abs().double()) + 2.0 ** -22 * (ref.abs() + bias.abs() + c0.abs())
    if layout == "nt":
        A, sa, B, sb = a.cuda(), (K, 1), b.T.contiguous().cuda(), (1, K)
    elif layout == "nn":
        A, sa, B, sb = a.cuda(), (K, 1), b.cuda(), (N, 1)
    elif layout == "tn":
        A, sa, B, sb = a.T.contiguous().cuda(), (1, M), b.cuda(), (N, 1)
    else:
        pad = 3 if layout == "odd stride" else 0
        sh = 1 if layout == "unaligned" else 0
        fa, fb = torch.zeros(M * (K + pad) + 4).cuda(), torch.zeros(K * (N + pad) + 4).cuda()
        A, B = fa[sh:], fb[sh:]
        A.as_strided((M, K), (K + pad, 1)).copy_(a)
        B.as_strided((K, N), (N + pad, 1)).copy_(b)
        sa, sb = (K + pad, 1), (N + pad, 1)
    ref, bound = ref.numpy(), bound.numpy()
    assert np.all(np.abs(_gemm(A, B, M, N, K, sa, sb) - ref) <= bound)
    got = _gemm(A, B, M, N, K, sa, sb, bias=bias.cuda(), relu=1)
    assert np.all(np.abs(got - np.maximum(ref + bias.double().numpy(), 0.0)) <= bound)
    got = _gemm(A, B, M, N, K, sa, sb, C=c0.cuda())
    assert np.all(np.abs(got - (ref + c0.double().numpy())) <= bound)


@pytest.mark.parametrize("rows,cols", [(1, 1), (31, 33), (33, 32), (2048, 1408)])
def test_training_column_sums(rows, cols):
    import ctypes
    import torch
    x = torch.randn(rows, cols, generator=torch.Generator().manual_seed(rows))
    d, out = x.cuda(), torch.zeros(cols, device="cuda")
    ab._check(ab.load_library().astcb200_train_colsum(ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(out.data_ptr()), rows, cols,
                                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    bound = rows * 2.0 ** -24 * x.abs().double().sum(0) + 1e-30
    assert bool(((out.cpu().double() - x.double().sum(0)).abs() <= bound).all())


@pytest.mark.parametrize("bx,by", [(4, 4), (8, 8), (10, 8), (12, 12)])
def test_extensions_with_and_without_kept_sums(bx, by):
    """Blocks of up to 64 texels keep the infill sums of a dual-plane candidate, larger ones do not."""
    w, h = bx * 7 - 2, by * 3
    img = synth.make_texture(w, h, 77)
    rng = np.random.default_rng(bx)
    img[:, :, 3] = rng.integers(0, 256, (h, w))  # an independent alpha: dual-plane blocks win
    img[:by, : 2 * bx] = (9, 200, 31, 40)        # two void-extent blocks
    enc = ab.ASTCEncoder(device=0, fixed=True, void_extent=True, dual_plane=True)
    enc.secondaryInit(w, h, bx, by)
    sym = enc.encode_symbolic(img)
    out = enc.encode(img).reshape(-1, 16)
    enc.close()
    orc = _libs.oracle()
    prev = orc.orc_set_extensions(3)
    try:
        ref_out, ref_sym = oracle_encode(img, bx, by, True)
    finally:
        orc.orc_set_extensions(prev)
    assert np.array_equal(sym, ref_sym)
    assert np.array_equal(out, ref_out)
    assert np.any(sym[:, 6] > 0) and np.any(sym[:, 7] > 0)


@pytest.mark.parametrize("bx,by", [(4, 4), (6, 6)])
@pytest.mark.parametrize("kmax,kbm", [(1, 1), (16, 5), (16, 50), (3, 64)])
def test_selection_among_equal_logits(bx, by, kmax, kbm):
    """Every partitioning and block mode with the same logit: more candidates than a warp collects,
    taken in class order."""
    from astc_implementation_b200 import proposal
    lay = proposal.Layout(bx, by)
    net = {"w1": np.zeros((256, lay.inputs)), "b1": np.zeros(256), "w2": np.zeros((256, 256)), "b2": np.zeros(256),
           "w3": np.zeros((lay.outputs, 256)), "b3": np.full(lay.outputs, 0.25)}
    enc = ab.ASTCEncoder(device=0, fixed=True)
    enc.set_proposal_net(net, bx, by)
    enc.set_pruning(True, max_partitionings=kmax, block_modes=kbm, coverage=1.0, threshold=0.0)
    w, h = 12 * bx, 9 * by - 1
    enc.secondaryInit(w, h, bx, by)
    route, picks, masks = enc.proposal_selection(synth.make_texture(w, h, 3))
    enc.close()
    assert np.all(route == 0) and np.all(picks[:, 0] == kmax)
    assert np.all(picks[:, 2:2 + kmax] == lay.pick_of(np.arange(kmax)))
    first = (1 << min(kbm, lay.nbm)) - 1
    for p in (0, 1):  # the single partition, and two partitions (the first classes)
        got = sum(masks[:, 4 * p + i].astype(object) << (64 * i) for i in range(4))
        assert np.all(got == first)


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("bx,by", [(4, 4), (8, 6)])
@pytest.mark.parametrize("blocks_x,blocks_y", [(227, 1),   # 2,951 partitioned blocks: 8 candidates a warp, four lanes each
                                               (12, 19),   # 2,964: 16, two lanes each
                                               (35, 13),   # 5,915: 16
                                               (24, 19)])  # 5,928: 32
def test_refinement_lanes_by_launch_size(bx, by, blocks_x, blocks_y, fixed):
    img = synth.make_texture(bx * blocks_x, by * blocks_y - 1, 83 + blocks_x)
    check_full_search(img, bx, by, fixed)


@pytest.mark.parametrize("bx,by", [(5, 5), (6, 6)])
def test_refinement_hands_over_by_launch_size(bx, by):
    """A launch of one wave keeps its candidates, one of a few waves hands most of them to the
    tail after the first iteration, a larger one the last of each group: the same blocks."""
    w, h = 100 * bx - 1, 46 * by - 2  # 4,600 blocks
    img = synth.make_texture(w, h, 71 + bx)
    outs, tails = [], []
    for chunk in (900, 1000, 0):
        enc = ab.ASTCEncoder(device=0, fixed=True, chunk_blocks=chunk, stage_timing=True)
        enc.secondaryInit(w, h, bx, by)
        outs.append(enc.encode(img).reshape(-1, 16))
        tails.append(int(enc.work_counters()[13]))
        enc.close()
    ref, _ = oracle_encode(img[:10 * by], bx, by, True)
    assert np.array_equal(outs[0][:1000], ref)
    assert np.array_equal(outs[1], outs[0]) and np.array_equal(outs[2], outs[0])
    assert tails[0] == 0 and tails[1] > tails[2] > 0


@pytest.mark.parametrize("bx,by", [(4, 4), (6, 6)])
@pytest.mark.parametrize("logit,route", [(-3.2e38, 1), (-2.0e38, 0)])
def test_selection_with_logits_near_the_lowest_value(bx, by, logit, route):
    """Below -3e38 no class counts, the softmax is 0 / 0 and the block takes the full search even at
    threshold 0; the places a lane holds beyond the last class must not stand in for one."""
    from astc_implementation_b200 import proposal
    lay = proposal.Layout(bx, by)
    net = {"w1": np.zeros((256, lay.inputs)), "b1": np.zeros(256), "w2": np.zeros((256, 256)), "b2": np.zeros(256),
           "w3": np.zeros((lay.outputs, 256)), "b3": np.full(lay.outputs, logit)}
    enc = ab.ASTCEncoder(device=0, fixed=True)
    enc.set_proposal_net(net, bx, by)
    enc.set_pruning(True, max_partitionings=2, block_modes=5, coverage=1.0, threshold=0.0)
    w, h = 12 * bx, 9 * by - 1
    enc.secondaryInit(w, h, bx, by)
    got, picks, _ = enc.proposal_selection(synth.make_texture(w, h, 3))
    enc.close()
    assert np.all(got == route)
    assert np.all(picks[:, 0] == (0 if route else 2))


@pytest.mark.parametrize("bx,by,blocks_x,blocks_y", [(6, 6, 46, 22),   # 1,012 blocks: 823 groups, little over one wave
                                                     (5, 5, 64, 71),   # 4,544: 3,692, little below five
                                                     (6, 6, 64, 72)])  # 4,608: 3,744, above: the last of each group only
def test_refinement_tail_takes_what_the_rule_offers(bx, by, blocks_x, blocks_y):
    """A launch of few waves offers the tail all of its candidates, which must have room for them; how many it
    takes does not depend on what the encoder encoded before."""
    img = synth.make_texture(bx * blocks_x - 1, by * blocks_y, 91)
    big = synth.make_texture(bx * 100, by * 100, 92)
    few = blocks_x * blocks_y <= 4553
    taken, outs = [], []
    for warm in (False, True):
        enc = ab.ASTCEncoder(device=0, fixed=True, stage_timing=True)
        if warm:
            enc.secondaryInit(big.shape[1], big.shape[0], bx, by)
            enc.encode(big)
        enc.secondaryInit(img.shape[1], img.shape[0], bx, by)
        outs.append(enc.encode(img))
        c = enc.work_counters()
        offered, accepted = int(c[13]), int(c[14])
        if few:
            assert accepted == offered > 30 * enc.numBlocks
        else:
            assert 0 < accepted <= min(offered, 16 * enc.numBlocks)
        taken.append(accepted)
        enc.close()
    assert np.array_equal(outs[0], outs[1])
    if few:
        assert taken[0] == taken[1]


@pytest.mark.parametrize("layout", ["nt", "nn", "tn", "odd stride", "unaligned"])
@pytest.mark.parametrize("M,N,K", [(1, 1, 16), (65, 63, 15), (2000, 900, 16),          # one slice, any number of tiles
                                   (33, 70, 17), (64, 64, 127), (2368, 768, 48),       # up to 444 tiles of 64x64
                                   (2369, 768, 48), (64, 64, 128), (200, 130, 1)])    # 456 tiles; split sums
def test_training_gemm_of_few_terms(M, N, K, layout):
    """Both sides of the small tiles' range, read along K and along the rows."""
    test_training_gemm_tiles_splits_and_layouts(M, N, K, layout)


@pytest.mark.parametrize("rows,cols", [(32, 4095), (32, 4096), (33, 4096), (1, 5000), (33, 32768), (128, 32769), (129, 32768)])
def test_training_column_sums_of_many_columns(rows, cols):
    """One thread a column or 32: the same partial sums, added in the same order."""
    import ctypes
    import torch
    x = torch.randn(rows, cols, generator=torch.Generator().manual_seed(rows))
    lib, s = ab.load_library(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    d, out, part = x.cuda(), torch.zeros(cols, device="cuda"), torch.zeros(64, device="cuda")
    ab._check(lib.astcb200_train_colsum(ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(out.data_ptr()), rows, cols, s))
    few = d[:, -64:].contiguous()  # 64 columns: 32 threads each
    ab._check(lib.astcb200_train_colsum(ctypes.c_void_p(few.data_ptr()), ctypes.c_void_p(part.data_ptr()), rows, 64, s))
    torch.cuda.synchronize()
    assert bool((out[-64:] == part).all())
    bound = rows * 2.0 ** -24 * x.abs().double().sum(0) + 1e-30
    assert bool(((out.cpu().double() - x.double().sum(0)).abs() <= bound).all())

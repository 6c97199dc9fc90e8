"""Device encodes without a stream: what waits for them and what does not."""
import time

import numpy as np
import pytest

import astc_implementation_b200 as ab
from astc_implementation_b200 import synth

pytestmark = pytest.mark.gpu

W, H, BX, BY = 1024, 512, 4, 4


@pytest.fixture(scope="module")
def job():
    """An encoder with a 10 ms search, its image, a second one and their blocks."""
    import torch
    enc = ab.ASTCEncoder(device=0)
    enc.secondaryInit(W, H, BX, BY)
    imgs = [synth.make_texture(W, H, 900 + i) for i in range(2)]
    blocks = [enc.encode(i) for i in imgs]
    dev = [torch.from_numpy(i.reshape(-1)).cuda() for i in imgs]
    out = torch.zeros(enc.numBlocks * 16, dtype=torch.uint8, device="cuda")
    enc.encode_device(dev[0].data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    yield enc, imgs, dev, out, blocks
    enc.close()


def queue(job, i, batch):
    """Encode i into `out`, which held the other image's blocks."""
    enc, _, dev, out, _ = job
    if batch:
        enc.encode_batch_device([(dev[i].data_ptr(), W, H, BX, BY, out.data_ptr(), out.numel())])
    else:
        enc.encode_device(dev[i].data_ptr(), out.data_ptr())


@pytest.mark.parametrize("batch", [False, True])
def test_other_default_stream_work_does_not_wait(job, batch):
    import torch
    default = torch.cuda.default_stream()
    queue(job, 0, batch)  # a batch's graph is captured by its first call
    torch.cuda.synchronize()
    ev = torch.cuda.Event()
    t0 = time.perf_counter()
    queue(job, 0, batch)
    ev.record(default)
    ev.synchronize()
    t_default = time.perf_counter() - t0
    torch.cuda.synchronize()
    t_all = time.perf_counter() - t0
    assert t_default < 0.5 * t_all


@pytest.mark.parametrize("batch", [False, True])
def test_readers_on_the_default_stream_wait(job, batch):
    import torch
    _, imgs, dev, out, blocks = job
    host = torch.zeros(16 + out.numel(), dtype=torch.uint8).pin_memory().numpy()
    texels = torch.zeros(W * H * 4, dtype=torch.uint8, device="cuda")
    sse = torch.zeros(4, dtype=torch.int64, device="cuda")
    for i in (1, 0, 1):
        queue(job, i, batch)
        ab.astc_containers_device([(out.data_ptr(), host, W, H, BX, BY)])
        torch.cuda.synchronize()
        assert np.array_equal(host[16:], blocks[i])
    ref = ab.decode(BX, BY, W, H, blocks[0])
    queue(job, 0, batch)
    ab.decode_device(BX, BY, W, H, out.data_ptr(), texels.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(texels.cpu().numpy().reshape(H, W, 4), ref)
    ref = ab.decode(BX, BY, W, H, blocks[1]).astype(np.int64) - imgs[1]
    queue(job, 1, batch)
    ab.decode_error_device(BX, BY, W, H, out.data_ptr(), dev[1].data_ptr(), sse.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(sse.cpu().numpy(), (ref * ref).reshape(-1, 4).sum(axis=0))


def test_encode_beside_a_capture(job):
    """A capture on another stream forbids the default stream; the encode does not touch it and leaves the
    capture valid."""
    import torch
    enc, _, dev, out, blocks = job
    x = torch.zeros(1 << 16, device="cuda")
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        x.add_(1.0)  # loaded before the capture
    torch.cuda.synchronize()
    out.zero_()
    torch.cuda.synchronize()
    x.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side, capture_error_mode="thread_local"):
        x.add_(1.0)
        enc.encode_device(dev[1].data_ptr(), out.data_ptr())
    g.replay()
    torch.cuda.synchronize()
    assert bool((x == 1.0).all())
    assert np.array_equal(out.cpu().numpy(), blocks[1])

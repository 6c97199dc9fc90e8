"""Launch counts reported by an encode (astcb200_stats.launches, astcb200_stage_times), against the kernels
its sequence queues."""
import numpy as np
import pytest

import astc_implementation_b200 as ab
from astc_implementation_b200 import proposal, synth

pytestmark = pytest.mark.gpu


def launches(w, h, bx, by, network, extend=False, chunk=0):
    enc = ab.ASTCEncoder(device=0, fixed=True, stage_timing=True, void_extent=extend, dual_plane=extend, chunk_blocks=chunk)
    if network:
        enc.set_proposal_net(proposal.load_weights(bx, by))
        enc.set_pruning(True)
    enc.secondaryInit(w, h, bx, by)
    enc.encode(synth.make_texture(w, h, 17))
    stages = enc.stage_times()[1].tolist()
    total = enc.last_stats.launches
    enc.close()
    return total, stages


# by stage: partition search and network, front, refinement, select-pack
@pytest.mark.parametrize("w,h,bx,by,extend,chunk,stages", [
    # 64 blocks: each pass's list is small whatever it holds, one refinement instance; the tail in the proposal pass
    (32, 32, 4, 4, False, 0, [3, 3, 3, 2]),
    # 1,500 blocks: both instances in each pass
    (200, 120, 4, 4, False, 0, [3, 3, 5, 2]),
    (200, 120, 4, 4, True, 0, [3, 3, 5, 2]),
    (200, 120, 4, 4, False, 1000, [6, 6, 9, 4]),  # the second chunk's 500 blocks: both in the fallback's 13 slots
    (300, 300, 6, 6, False, 0, [3, 3, 5, 2]),
    # 20 x 2 of 10x8: no tail above 36 texels, no network: the full search
    (200, 16, 10, 8, False, 0, [1, 1, 1, 1]),
])
def test_launch_counts(w, h, bx, by, extend, chunk, stages):
    total, got = launches(w, h, bx, by, (bx, by) in ((4, 4), (6, 6)), extend, chunk)
    assert got == stages
    assert total == sum(stages) + (1 if extend else 0)


@pytest.mark.parametrize("w,h,refine", [(400, 300, 2),        # 7,500 blocks: more than one wave, with a tail
                                        (4 * 911, 4, 2),      # 741 groups of 16 partitioned blocks: as few as have one
                                        (4 * 910, 4, 1),      # 740: one wave hands nothing over and has none
                                        (64, 64, 1)])
def test_launch_counts_of_a_full_search(w, h, refine):
    total, got = launches(w, h, 4, 4, False)
    assert got == [1, 1, refine, 1] and total == 3 + refine


def test_launch_counts_of_a_batch():
    """A batch of one texture queues the texture's own sequence."""
    enc = ab.ASTCEncoder(device=0, fixed=True)
    enc.set_proposal_net(proposal.load_weights(4, 4))
    enc.set_pruning(True)
    img = synth.make_texture(200, 120, 17)
    enc.encode_batch([(img, 4, 4)])
    assert enc.last_stats.launches == 13
    enc.close()

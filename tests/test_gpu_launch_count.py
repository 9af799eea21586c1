"""GPU: fa_kernel_launches counts what a solve launches. A round of a solve is the pass, in one form (at
most 592 work items, or more) or both where the list may need either, the reduction of its own for
frames of more than 2048 tiles, and the step. What a solve launches besides its rounds is known, so the
count less that has to be a multiple of a round."""
import numpy as np
import pytest

import fa_b200 as fa
import fa_synth as S

pytestmark = pytest.mark.gpu

BURST = 4  # iterations that a single-frame solve queues, and that a batch's graph holds


def _frames(shape, nD, n, tile_voxels):
    ok, msg = fa.gpu_support()
    assert ok, msg
    nz, ny, nx = shape
    acq = S.make_acquisition(shape, nD, 1, S.BlobSpec(60, (2.0, 6.0), (1.0, 2.0), mean=30.0),
                             S.WalkSpec(1.0, 3.0, 0.0, 0.0), seed=9)
    line, il, ifr = acq.scan
    ref = fa.Reference(fa.Context(), acq.reference + 1, nD, fa.scan_params(line, il, ifr, nx, ny, nz))
    ref.retune(tile_voxels, 2)
    tiles = -(-nz * ny // max(1, tile_voxels // nx))
    return [fa.Frame(ref, acq.frames[0] + 1) for _ in range(n)], tiles


# tile rows of 16, 1 and 1: 16, 256 and 4096 tiles a frame
@pytest.mark.parametrize("shape,nD,tile,kernels", [((1, 256, 256), 8, 4096, 2), ((8, 512, 128), 16, 128, 3),
                                                   ((8, 512, 129), 16, 129, 3)],
                         ids=["few", "wide", "wide, odd rows"])
def test_single_frame_solve(shape, nD, tile, kernels):
    (frame,), tiles = _frames(shape, nD, 1, tile)
    assert (tiles > 2048) == (kernels == 3)
    before = fa.kernel_launches()
    frame.align(None, 2)
    n = fa.kernel_launches() - before - 1  # the start
    assert n > 0 and n % (BURST * kernels) == 0 and n // (BURST * kernels) <= 2


@pytest.mark.parametrize("shape,nD,tile,n,kernels", [((1, 256, 256), 8, 4096, 2, 2), ((1, 256, 256), 8, 256, 4, 3),
                                                     ((8, 512, 128), 16, 128, 2, 3), ((8, 512, 129), 16, 129, 2, 3)],
                         ids=["few", "both forms", "wide", "wide, odd rows"])
def test_batched_solve(shape, nD, tile, n, kernels):
    frames, tiles = _frames(shape, nD, n, tile)
    before = fa.kernel_launches()
    fa.align_batch(frames, None, 2)
    count = fa.kernel_launches() - before - 1  # the first list
    assert count > 0 and count % (BURST * kernels) == 0 and count // (BURST * kernels) <= 2

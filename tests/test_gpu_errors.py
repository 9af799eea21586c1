"""GPU: a call that CUDA refuses reports its error once; the same thread's next calls are fine."""
import numpy as np
import pytest

import fa_b200 as fa
import fa_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 64, 64), (1, 61, 37), (8, 256, 256)], ids=lambda s: "x".join(map(str, s)))
def test_a_refused_call_does_not_fail_the_next(shape):
    ok, msg = fa.gpu_support()
    assert ok, msg
    nz, ny, nx = shape
    acq = S.make_acquisition(shape, 10, 1, S.BlobSpec(30, (2.0, 6.0), (1.0, 2.0), mean=30.0),
                             S.WalkSpec(1.0, 3.0, 0.0, 0.0), seed=3)
    line, il, ifr = acq.scan
    ctx = fa.Context()
    ref = fa.Reference(ctx, acq.reference + 1, acq.nD, fa.scan_params(line, il, ifr, nx, ny, nz))
    frame = fa.Frame(ref, acq.frames[0] + 1)
    corr = fa.Correlator(ctx, acq.reference)
    D = acq.D_true[0]
    calls = [lambda: frame.warp(D), lambda: frame.get_error(D), lambda: frame.align(None, 3)[0],
             lambda: corr.compute_shift(acq.frames[0]), lambda: fa.align_batch([frame], None, 3)[0],
             lambda: ref.warp_image(acq.frames[0], D)[0].shape]  # (a splat by atomics: its last bits vary)
    for call in calls:
        want = call()
        with pytest.raises(fa.FaError):
            fa.Context(device=4711)  # no such device
        assert np.array_equal(call(), want)

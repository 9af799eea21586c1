"""GPU: the phase correlator's last step (first maximum over the row pass's partial maxima) and its
batches, at the edges of its block sizes.

The peak is a whole number and has to be the surface's first maximum exactly; equal values (a zero
frame) and a surface without a maximum (NaN) give index 0, as a strict `>` from -DBL_MAX does. A
batch's results are those of single-frame calls, bit for bit: batches are cut at 64 frames.
"""
import numpy as np
import pytest

import fa_b200 as fa

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    ok, msg = fa.gpu_support()
    assert ok, msg
    return fa.Context()


# partial maxima per frame: few, 512, 1024 and 2048 (one block of 256 threads takes up to 1024 pairs)
@pytest.mark.parametrize("shape", [(1, 8, 16), (16, 512, 512), (32, 512, 512), (64, 512, 512)],
                         ids=lambda s: "x".join(map(str, s)))
def test_peak_is_the_surface_first_maximum(ctx, shape):
    nz, ny, nx = shape
    rng = np.random.default_rng(nz + nx)
    ref = rng.integers(0, 1000, shape).astype(np.float32)
    c = fa.Correlator(ctx, ref)
    for shift in ((0, 0, 0), (-1 % nz, -1, -1), (nz // 2, 3, 2), (0, -2, 4)):
        vol = np.roll(ref, shift, axis=(0, 1, 2))
        idx = np.unravel_index(int(np.argmax(c.surface(vol, planes=True))), shape)
        want = [v - n if v > n // 2 else v for v, n in zip(idx[::-1], (nx, ny, nz))]
        assert np.array_equal(c.compute_shift(vol), np.array(want, np.float64))
    assert np.array_equal(c.compute_shift(np.zeros(shape, np.float32)), np.zeros(3))
    assert np.array_equal(c.compute_shift(np.full(shape, np.nan, np.float32)), np.zeros(3))
    c.close()


@pytest.mark.parametrize("shape", [(1, 32, 64), (2, 30, 36)], ids=["planes", "cufft"])
@pytest.mark.parametrize("frames", [63, 65, 130])
def test_batches_equal_single_frames(ctx, shape, frames):
    rng = np.random.default_rng(frames)
    ref = (rng.random(shape) * 1000).astype(np.float32)
    vols = [np.roll(ref, (0, int(rng.integers(-3, 4)), int(rng.integers(-3, 4))), axis=(0, 1, 2)).astype(np.uint16)
            for _ in range(frames)]
    import torch

    dev = [torch.from_numpy(v.view(np.int16)).cuda() for v in vols]
    torch.cuda.synchronize()
    ptrs = [d.data_ptr() for d in dev]
    a = fa.Aligner(ctx, nD=4, precision=fa.PREC_MIXED, max_iterations=2)
    nz, ny, nx = shape
    a.set_reference(ref, fa.scan_params(1.0, 1.01, ny * 1.01, nx, ny, nz))
    D, _ = a.add_frames_device(ptrs, fa.U16, frames)
    for i in (0, 1, 62, 63 % frames, frames - 1):
        one, _ = a.add_frames_device(ptrs[i:i + 1], fa.U16, 1)
        assert np.array_equal(D[i], one[0])
    a.close()

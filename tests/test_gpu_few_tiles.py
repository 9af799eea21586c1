"""GPU: the fused pass's forms for few tiles (csrc/fa_eval4.cu, eval4_tile_cta: one tile per CTA, errors
by all warps, then the summation chains; csrc/fa_kernels.cu, eval_kernel in runs, for rows that are no
multiple of four voxels) at the edges of their range, and the first against the one-warp-per-tile form,
whose partial sums it has to reproduce bit for bit.

Tolerances, against the FP64 statement of one evaluation on the values the device stores
(oracle_py.fp64_error_jacobian): the summation bounds of test_gpu_mixed.py, f relative 5e-6 and J^T e
5e-5 of max|J^T e| -- both forms sum a lane's at most 128 terms of a tile in FP32 and the rest pairwise
-- with mixed storage, and 2e-6 / 2e-5 with FP32 storage."""
import numpy as np
import pytest

import fa_b200 as fa
import fa_synth as S
import oracle_py as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    ok, msg = fa.gpu_support()
    assert ok, msg
    return fa.Context()


def _acq(shape, nD, n_frames=1):
    nz = shape[0]
    return S.make_acquisition(shape, nD, n_frames,
                              S.BlobSpec(int(200 * shape[1] * shape[2] / 65536) + 20, (2.0, 6.0), (1.0, 2.0), mean=30.0),
                              S.WalkSpec(1.0, 4.0, 0.3 if nz > 1 else 0.0, 1.0 if nz > 1 else 0.0), seed=41)


# rows of 4 (one lane of a segment) and 8, of a segment and a little more, of several segments; tiles of
# more than 32 segments (narrow rows: several batches), of fewer than 32 (short volumes, one warp's
# worth), a last tile that is cut, one range per tile and two
SHAPES = [((1, 64, 4), 4), ((1, 700, 8), 5), ((1, 96, 128), 6), ((1, 70, 132), 5), ((1, 33, 1028), 4),
          ((2, 40, 64), 6), ((5, 61, 100), 10), ((3, 37, 256), 7), ((16, 24, 384), 32),
          # rows that are no multiple of four: shorter than a step of 32 voxels, of one, of four and a little more
          ((1, 64, 5), 4), ((1, 300, 33), 5), ((1, 70, 127), 6), ((1, 90, 129), 6), ((5, 61, 103), 10), ((3, 37, 257), 7)]


@pytest.mark.parametrize("precision", [fa.PREC_F32, fa.PREC_MIXED], ids=["f32", "mixed"])
@pytest.mark.parametrize("bidirectional", [False, True], ids=["uni", "bidi"])
@pytest.mark.parametrize("shape,nD", SHAPES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_evaluation_matches_fp64_statement(ctx, shape, nD, bidirectional, precision):
    acq = _acq(shape, nD)
    nz, ny, nx = shape
    line, il, ifr = acq.scan
    ref_p1 = acq.reference + 1
    frame = (acq.frames[0] + 1).astype(np.float32)
    ow = O.OracleWarper(ref_p1, nD, O.scan_init(line, il, ifr, nx, ny, nz, bidirectional))
    ref = fa.Reference(ctx, ref_p1, nD, fa.scan_params(line, il, ifr, nx, ny, nz, bidirectional), precision)
    fr = fa.Frame(ref, frame)
    grad = ow.gradient()
    stored = (ref_p1, grad, frame)
    tol_f, tol_g = 2e-6, 2e-5
    if precision == fa.PREC_MIXED:
        stored = (O.round_bf16(ref_p1), [O.round_bf16(g) for g in grad], frame.astype(np.float16).astype(np.float32))
        tol_f, tol_g = 5e-6, 5e-5
    rng = np.random.Generator(np.random.PCG64(3))
    # at rest, near the truth, and far enough that windows leave the halo on every side
    for D in (np.zeros((nD, 3)), acq.D_true[0] + rng.normal(0, 0.3, (nD, 3)), rng.uniform(-0.3, 0.3, (nD, 3)) * [nx, ny, nz]):
        if nz == 1:
            D[:, 2] = 0.0
        f64, g64 = O.fp64_error_jacobian(ow, *stored, D)
        f, g = fr.get_error(D), fr.get_jacobian(D)
        assert abs(f - f64) <= tol_f * f64
        assert np.max(np.abs(g - g64)) <= tol_g * np.max(np.abs(g64))
    fr.close()
    ref.close()


@pytest.mark.parametrize("shape,nD,n", [((1, 512, 512), 16, 16), ((8, 132, 260), 16, 20)])
def test_same_solves_as_the_form_for_many_tiles(ctx, shape, nD, n):
    """Frames solved together start in the one-warp-per-tile form (more than 592 items) and end in the
    other; alone they stay in the other. Their displacements are identical."""
    acq = _acq(shape, nD, 4)
    nz, ny, nx = shape
    line, il, ifr = acq.scan
    ref = fa.Reference(ctx, acq.reference + 1, nD, fa.scan_params(line, il, ifr, nx, ny, nz), fa.PREC_MIXED)
    frames = [fa.Frame(ref, acq.frames[k % 4] + 1) for k in range(n)]
    rigid = np.array([np.round(acq.D_true[k % 4].mean(0)) for k in range(n)])
    assert n * -(-nz * ny // max(1, 4096 // nx)) > 592
    D, _ = fa.align_batch(frames, rigid, 100)
    for k in range(4):
        assert np.array_equal(D[k], frames[k].align(rigid[k], 100)[0])
        for j in range(k + 4, n, 4):
            assert np.array_equal(D[j], D[k])
    for f in frames:
        f.close()
    ref.close()

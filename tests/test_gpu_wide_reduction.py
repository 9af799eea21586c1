"""GPU: the reduction of tile sums over many CTAs (csrc/fa_kernels.cu, wide_reduce_kernel), which bare
evaluations of more than 768 tiles and solves of more than 2048 take.

Its sums are those of the one-CTA form and of the order stated here, bit for bit: f in 128 strided runs and
a fixed tree, g tile by tile in FP64. A frame solved together with frames of the other form gives
what it gives alone, bit for bit, and a served one what the aligner gives (1e-9 px, as in
test_gpu_server.py)."""
import numpy as np
import pytest

import fa_b200 as fa
import fa_synth as S

pytestmark = pytest.mark.gpu

PARTIAL = 12


@pytest.fixture(scope="module")
def ctx():
    ok, msg = fa.gpu_support()
    assert ok, msg
    return fa.Context()


def _ordered(c0, parts, nD, n_dim):
    runs = np.zeros(128)
    for t in range(len(c0)):  # run t % 128, ascending
        runs[t % 128] += parts[t, 0]
    w = 64
    while w:
        runs[:w] = runs[:w] + runs[w:2 * w]
        w //= 2
    g = np.zeros((nD, n_dim))
    for t in range(len(c0)):
        for s in range(3):
            if c0[t] + s < nD:
                g[c0[t] + s] += parts[t, 2 + 3 * s:2 + 3 * s + n_dim]
    return np.concatenate([runs[:1], g.ravel()])


# a tile or two, all tiles in one range, ends of a stage of 512 tiles, many ranges, the most tiles of a large volume
@pytest.mark.parametrize("n_tiles,nD", [(1, 2), (2, 3), (127, 4), (513, 3), (1024, 2), (1536, 40), (2049, 7), (4100, 300),
                                        (16384, 64)])
@pytest.mark.parametrize("n_dim", [2, 3])
def test_both_forms_keep_the_order(ctx, n_tiles, nD, n_dim):
    rng = np.random.default_rng(n_tiles + nD)
    c0 = np.sort(rng.integers(0, nD - 1, n_tiles)).astype(np.int32)
    parts = rng.standard_normal((n_tiles, PARTIAL)) * 10.0 ** rng.integers(-6, 7, (n_tiles, PARTIAL))
    parts[c0 == nD - 2, 8:11] = 0.0  # no control point nD
    want = _ordered(c0, parts, nD, n_dim)
    assert np.array_equal(fa.test_reduce(ctx, nD, n_dim, c0, parts, False), want)
    assert np.array_equal(fa.test_reduce(ctx, nD, n_dim, c0, parts, True), want)


def _frame(ctx, shape, nD, tile_voxels, seed):
    nz, ny, nx = shape
    acq = S.make_acquisition(shape, nD, 1, S.BlobSpec(80, (2.0, 6.0), (1.0, 2.0), mean=30.0),
                             S.WalkSpec(1.0, 4.0, 0.3 if nz > 1 else 0.0, 1.0 if nz > 1 else 0.0), seed=seed)
    line, il, ifr = acq.scan
    ref = fa.Reference(ctx, acq.reference + 1, nD, fa.scan_params(line, il, ifr, nx, ny, nz), fa.PREC_MIXED)
    ref.retune(tile_voxels, 2)
    return fa.Frame(ref, acq.frames[0] + 1), np.round(acq.D_true[0].mean(0)), acq


# 1024 tiles: the evaluation takes the wide form, the solve's steps the other; 2100: both the wide one
@pytest.mark.parametrize("shape,tile", [((1, 1024, 64), 64), ((1, 1024, 65), 65), ((5, 420, 64), 64), ((5, 420, 65), 65)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_evaluation_equals_the_solve_s_value(ctx, shape, tile):
    frame, rigid, acq = _frame(ctx, shape, 12, tile, 31)
    D, stats = frame.align(rigid, 100)
    assert frame.get_error(D) == stats["f_final"]
    frame.update(acq.frames[0] + 1)
    assert frame.get_error(D) == stats["f_final"]


@pytest.mark.parametrize("nx", [64, 65])
def test_batch_of_both_forms_equals_single_solves(ctx, nx):
    made = [_frame(ctx, (5, 420, nx), 12, nx, 32), _frame(ctx, (2, 200, nx), 12, nx, 33),
            _frame(ctx, (5, 450, nx), 12, nx, 34)]  # 2100, 400 and 2250 tiles
    frames, rigid = [m[0] for m in made], np.array([m[1] for m in made])
    alone = [f.align(r, 100) for f, r in zip(frames, rigid)]
    D, stats = fa.align_batch(frames, rigid, 100)
    for k, (D1, s1) in enumerate(alone):
        assert np.array_equal(D[k], D1), k
        assert stats[k]["f_final"] == s1["f_final"] and stats[k]["iterations"] == s1["iterations"]


@pytest.mark.parametrize("nx", [4100, 4125])
def test_served_frames_of_many_tiles(ctx, nx):
    shape, nD = (9, 256, nx), 20  # 2304 rows, one to a tile
    acq = S.make_acquisition(shape, nD, 2, S.BlobSpec(400, (2.0, 6.0), (1.0, 2.0), mean=20.0),
                             S.WalkSpec(1.0, 3.0, 0.3, 1.0), seed=35)
    line, il, ifr = acq.scan
    scan = fa.scan_params(line, il, ifr, nx, 256, 9)
    raw = np.ascontiguousarray(acq.frames.astype(np.uint16))
    al = fa.Aligner(ctx, nD=nD, precision=fa.PREC_MIXED)
    al.set_reference(acq.reference, scan)
    D, _ = al.add_frames([raw[0], raw[1]])
    al.close()
    srv = fa.Server(ctx, warm_start=False)
    a = srv.add_acquisition(acq.reference, scan, frame_dtype=np.uint16, nD=nD, precision=fa.PREC_MIXED)
    tickets = [srv.submit(a, raw[k]) for k in range(2)]
    served = [srv.wait(t, 120.0)[0] for t in tickets]
    srv.close()
    for k in range(2):
        assert np.max(np.abs(served[k] - D[k])) <= 1e-9

"""GPU: host threads that call the library at the same time, each on handles of its own, with kernels
whose shared memory depends on the sizes: every call succeeds and returns what it returns alone. (The
permission for more than 48 KB is the process's, so a launch must not depend on what another
thread asked for last.)"""
import threading

import numpy as np
import pytest

import fa_b200 as fa
import fa_synth as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    ok, msg = fa.gpu_support()
    assert ok, msg
    return fa.Context()


def _acq(shape, nD):
    nz = shape[0]
    return S.make_acquisition(shape, nD, 1, S.BlobSpec(60, (2.0, 6.0), (1.0, 2.0), mean=30.0),
                              S.WalkSpec(1.0, 4.0, 0.3 if nz > 1 else 0.0, 1.0 if nz > 1 else 0.0), seed=17)


def _frame(ctx, acq, precision=fa.PREC_F32):
    nz, ny, nx = acq.reference.shape
    line, il, ifr = acq.scan
    ref = fa.Reference(ctx, acq.reference + 1, acq.nD, fa.scan_params(line, il, ifr, nx, ny, nz), precision)
    return fa.Frame(ref, acq.frames[0] + 1)


def _at_once(calls, rounds):
    """Each call in a thread of its own, `rounds` times; the first result of each, alone, is what every
    later one has to be."""
    want = [c() for c in calls]
    start, failed = threading.Barrier(len(calls)), []

    def run(call, expected):
        start.wait()
        try:
            for _ in range(rounds):
                got = call()
                assert np.array_equal(got, expected, equal_nan=True)
        except BaseException as e:  # noqa: BLE001 -- reported by the caller
            failed.append(e)

    threads = [threading.Thread(target=run, args=cw) for cw in zip(calls, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def test_solves_of_different_control_point_counts(ctx):
    """Steps that stage 41, 100 and 150 KB."""
    acqs = [_acq((16, 128, 128), nD) for nD in (67, 161, 240)]
    frames = [_frame(ctx, a) for a in acqs]
    rigid = [np.round(a.D_true[0].mean(0)) for a in acqs]
    _at_once([lambda f=f, r=r: f.align(r, 2)[0] for f, r in zip(frames, rigid)], 400)


def test_solves_of_one_size(ctx):
    """Several frames of one reference: passes and steps whose launches overlap their predecessors'."""
    acq = _acq((1, 256, 256), 16)
    frames = [_frame(ctx, acq) for _ in range(4)] + [_frame(ctx, acq, fa.PREC_MIXED)]
    rigid = np.round(acq.D_true[0].mean(0))
    _at_once([lambda f=f: f.align(rigid, 100)[0] for f in frames], 200)
    _at_once([lambda f=f: fa.align_batch([f], rigid[None], 100)[0] for f in frames], 20)


def test_warps_of_different_control_point_counts(ctx):
    """57 and 91 KB of control-point parameters."""
    acqs = [_acq((1, 2048, 16), nD) for nD in (1200, 1900)]
    frames = [_frame(ctx, a) for a in acqs]
    _at_once([lambda f=f, a=a: f.warp(a.D_true[0]) for f, a in zip(frames, acqs)], 400)


@pytest.mark.parametrize("shapes", [((1, 64, 64), (1, 2048, 64)), ((1, 16, 2048), (1, 16, 4096)),
                                    ((32, 16, 64), (32, 1024, 16))], ids=["yz", "rows", "split"])
def test_correlations_of_different_sizes(ctx, shapes):
    import torch

    rng = np.random.default_rng(5)
    calls = []
    for shape in shapes:
        ref = (rng.random(shape) * 1000).astype(np.float32)
        vol = torch.from_numpy(np.roll(ref, (0, 3, -2), axis=(0, 1, 2)).copy()).cuda()
        corr = fa.Correlator(ctx, ref)
        calls.append(lambda c=corr, v=vol: c.compute_shift_device(v.data_ptr()))
    torch.cuda.synchronize()
    _at_once(calls, 600)

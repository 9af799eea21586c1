"""GPU: the solve graphs an aligner keeps. A call whose groups it has had before captures nothing, also
when calls of other groups came between (host and device frames in turn, another number of
frames); how many are kept is bounded, and a range that was given up is solved like any other."""
import numpy as np
import pytest

import fa_b200 as fa
import fa_synth as S

pytestmark = pytest.mark.gpu


def _aligner(shape, nD, seed):
    ok, msg = fa.gpu_support()
    assert ok, msg
    nz, ny, nx = shape
    acq = S.make_acquisition(shape, nD, 2, S.BlobSpec(100, (2.0, 6.0), (1.0, 2.0), mean=20.0),
                             S.WalkSpec(1.0, 3.0, 0.3 if nz > 1 else 0.0, 1.0 if nz > 1 else 0.0), seed=seed)
    line, il, ifr = acq.scan
    al = fa.Aligner(fa.Context(), nD=nD, precision=fa.PREC_MIXED)
    al.set_reference(acq.reference, fa.scan_params(line, il, ifr, nx, ny, nz))
    return al, np.ascontiguousarray(acq.frames.astype(np.uint16))


def _calls(al, raw):
    import torch

    dev = torch.from_numpy(raw.view(np.int16)).to("cuda:0")
    torch.cuda.synchronize()
    host = lambda n: al.add_frames([raw[k % 2] for k in range(n)])[0]  # noqa: E731
    device = lambda n: al.add_frames_device([dev[k % 2].data_ptr() for k in range(n)], fa.U16, n)[0]  # noqa: E731
    return host, device, dev


def test_calls_in_turn_capture_once():
    al, raw = _aligner((16, 512, 512), 16, 71)  # 8.4 MB a frame: groups of 4 from the host, of 8 from the device
    host, device, _dev = _calls(al, raw)
    turn = [(host, 16), (device, 16), (host, 15), (device, 13), (host, 3)]
    first = [f(n) for f, n in turn]
    captured, kept = al.graphs()
    assert kept == captured > 0
    for _ in range(2):
        for (f, n), want in zip(turn, first):
            assert np.array_equal(f(n), want)
    assert al.graphs() == (captured, kept)
    al.close()


def test_graphs_kept_are_bounded():
    al, raw = _aligner((1, 32, 64), 4, 72)
    _host, device, _dev = _calls(al, raw)
    want = device(200)
    for n in range(199, 40, -1):  # the last group's range is another in most of these calls
        assert np.array_equal(device(n), want[:n]), n
    captured, kept = al.graphs()
    assert captured > 128 and kept <= 128
    assert np.array_equal(device(200), want)
    assert al.graphs()[1] <= 128
    al.close()


def test_kept_graphs_do_not_exhaust_the_budget():
    """With the smallest memory budget that a call of 40 frames fits, calls of fewer frames fit too: what is
    kept for other ranges is given back."""
    import torch

    shape, nD = (1, 32, 64), 4
    acq = S.make_acquisition(shape, nD, 2, S.BlobSpec(40, (2.0, 6.0), (1.0, 2.0), mean=20.0),
                             S.WalkSpec(1.0, 3.0, 0.0, 0.0), seed=73)
    line, il, ifr = acq.scan
    dev = torch.from_numpy(np.ascontiguousarray(acq.frames.astype(np.uint16)).view(np.int16)).to("cuda:0")
    torch.cuda.synchronize()

    def aligner(budget):
        al = fa.Aligner(fa.Context(memory_budget=budget), nD=nD, precision=fa.PREC_MIXED)
        al.set_reference(acq.reference, fa.scan_params(line, il, ifr, 64, 32, 1))
        return al

    def call(al, n):
        return al.add_frames_device([dev[k % 2].data_ptr() for k in range(n)], fa.U16, n)[0]

    def fits(budget):
        try:
            call(aligner(budget), 40)
            return True
        except fa.FaError as e:
            assert e.status == fa.FA_ERR_OOM
            return False

    lo, hi = 1 << 12, 1 << 28
    assert fits(hi)
    while hi - lo > 64:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if fits(mid) else (mid, hi)
    al = aligner(hi)
    want = call(al, 40)
    for n in (39, 36, 33, 20, 7, 1, 40, 12, 40):
        assert np.array_equal(call(al, n), want[:n]), n
    al.close()

"""GPU: the first call on new frame slots. A slot is cleared (its halo has to be zeros) before the streams that
fill it get to it, so a new aligner's first call, and a new server's, give what the second gives."""
import numpy as np
import pytest

import fa_b200 as fa
import fa_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [fa.PREC_F32, fa.PREC_MIXED], ids=["f32", "mixed"])
def test_first_call_equals_the_second(precision):
    import torch

    ok, msg = fa.gpu_support()
    assert ok, msg
    shape, nD, n = (16, 1024, 512), 16, 3  # slots of 34 or 17 MB
    acq = S.make_acquisition(shape, nD, n, S.BlobSpec(300, (2.0, 6.0), (1.0, 2.0), mean=20.0),
                             S.WalkSpec(1.0, 3.0, 0.3, 1.0), seed=81)
    line, il, ifr = acq.scan
    scan = fa.scan_params(line, il, ifr, shape[2], shape[1], shape[0])
    dev = torch.from_numpy(np.ascontiguousarray(acq.frames, np.float32)).to("cuda:0")
    torch.cuda.synchronize()
    ptrs = [dev[k].data_ptr() for k in range(n)]
    ctx = fa.Context()
    want = None
    for _ in range(3):
        al = fa.Aligner(ctx, nD=nD, precision=precision)
        al.set_reference(acq.reference, scan)
        first = al.add_frames_device(ptrs, fa.F32, n)[0]
        assert np.array_equal(first, al.add_frames_device(ptrs, fa.F32, n)[0])
        assert want is None or np.array_equal(first, want)
        want = first
        al.close()
        srv = fa.Server(ctx, warm_start=False)
        a = srv.add_acquisition(acq.reference, scan, frame_dtype=np.float32, nD=nD, precision=precision)
        served = [srv.wait(srv.submit_ptr(a, p, True), 120.0)[0] for p in ptrs + ptrs]
        for k in range(2 * n):
            assert np.max(np.abs(served[k] - want[k % n])) <= 1e-9  # as in test_gpu_server.py
        srv.close()

"""GPU: the solve groups of a call on host frames (csrc/fa_api.cu, host_group_frames): 8 frames where a
frame uploads quickly, 4 and 2 where it does not, the last group halved. Frames are independent and each
one's sums have a fixed order, so for any number of frames the displacements are those of the same
frames in device memory, bit for bit."""
import numpy as np
import pytest

import fa_b200 as fa
import fa_synth as S

pytestmark = pytest.mark.gpu

# 2 MB (groups of 8), 8.4 MB (4), 16.8 MB (2) and 33.6 MB (2: more than a group's upload) a frame
CASES = [((4, 512, 512), np.uint16, (1, 8, 9, 13)), ((16, 512, 512), np.uint16, (1, 2, 3, 5, 7, 8)),
         ((16, 512, 512), np.float32, (1, 2, 3, 4, 5)), ((8, 1024, 1024), np.float32, (1, 2, 3))]


@pytest.mark.parametrize("shape,dtype,counts", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v.__name__)
def test_host_groups_equal_device_frames(shape, dtype, counts):
    import torch

    ok, msg = fa.gpu_support()
    assert ok, msg
    nz, ny, nx = shape
    acq = S.make_acquisition(shape, 16, 2, S.BlobSpec(400, (2.0, 6.0), (1.0, 2.0), mean=20.0),
                             S.WalkSpec(1.0, 3.0, 0.3, 1.0), seed=61)
    line, il, ifr = acq.scan
    al = fa.Aligner(fa.Context(), nD=acq.nD, precision=fa.PREC_MIXED)
    al.set_reference(acq.reference, fa.scan_params(line, il, ifr, nx, ny, nz))
    host = np.ascontiguousarray(acq.frames.astype(dtype))
    dev = torch.from_numpy(host.view(np.int16) if dtype == np.uint16 else host).to("cuda:0")
    torch.cuda.synchronize()
    for n in counts:
        D, _ = al.add_frames([host[k % 2] for k in range(n)])
        D_dev, _ = al.add_frames_device([dev[k % 2].data_ptr() for k in range(n)],
                                        fa.U16 if dtype == np.uint16 else fa.F32, n)
        assert np.array_equal(D, D_dev), n
    al.close()

"""CPU: the launch of the one-kernel (z, y) pass (csrc/fa_plane_corr.cu, plane_yz_launch, which the launcher
uses too): a CTA's planes are the points its threads hold, every plane has one, and two CTAs fit an SM."""
import pytest

import fa_b200 as fa

POINTS = 4096  # 256 threads of 16 points


@pytest.mark.parametrize("nz", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("ny", [8, 16, 64, 128, 256, 512, 1024, 2048])
@pytest.mark.parametrize("nx,batch", [(16, 1), (64, 3), (512, 64)])
def test_one_kernel_pass(nz, ny, nx, batch):
    if nz * ny > 2 * POINTS:
        with pytest.raises(fa.FaError):  # split
            fa.plane_launch(nz, ny, nx, batch)
        return
    planes, ctas, smem = fa.plane_launch(nz, ny, nx, batch)
    n = batch * (nx // 2 + 1)
    if nz * ny == 2 * POINTS:  # a pair of CTAs, half of the z lines each
        assert planes == 0 and ctas == 2 * n
        lines = nz // 2
    else:
        assert planes >= 1 and planes * nz * ny <= POINTS < (planes + 1) * nz * ny
        assert (ctas - 1) * planes < n <= ctas * planes
        lines = planes * nz
    assert smem == 16 * (lines * (ny + 1) + ny)
    assert 2 * (smem + 1024) <= 228 * 1024  # (a CTA's system share is 1 KB)


@pytest.mark.parametrize("shape", [(3, 20, 30), (32, 16, 16), (1, 4, 64)])
def test_other_dimensions(shape):
    with pytest.raises(fa.FaError):
        fa.plane_launch(*shape, 1)

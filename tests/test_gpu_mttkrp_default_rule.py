"""CUD_PREC_DEFAULT takes the faster of the tensor cores and plain FP32 (which is
the more accurate one, and keeps ties): the kernel that cud_mttkrp_path names
where both were timed on B200, us a mode."""
import pytest

pytestmark = pytest.mark.gpu

TIMED = [  # dims, mode, R, tensor cores, FP32
    ((128, 128, 128), 0, 32, 12.1, 10.9), ((128, 128, 128), 1, 48, 13.5, 15.2), ((160, 160, 160), 1, 12, 14.3, 13.8),
    ((256, 256, 256), 0, 4, 20.8, 14.7), ((160, 160, 160), 2, 32, 16.6, 21.3), ((512, 512, 512), 0, 64, 120., 424.),
    # few rows of the mode: both compute whole tiles of 128
    ((256, 4, 256), 1, 64, 16.2, 34.9), ((256, 4, 256), 1, 32, 18.4, 21.3), ((256, 4, 256), 1, 8, 15.4, 12.3),
    ((512, 64, 8), 2, 64, 12.3, 22.9),
    ((1024, 1, 1024), 1, 16, 88., 130.),
    # Khatri-Rao rows built per stage
    ((200, 200, 200), 1, 16, 52., 22.), ((700, 5, 700), 1, 32, 361., 119.), ((3, 256, 256, 32), 2, 16, 42., 72.),
    ((3, 256, 256, 32), 3, 16, 117., 196.), ((256, 3, 256, 32), 0, 16, 43., 50.), ((2, 2, 1000, 1000), 3, 8, 23., 61.),
    ((6, 100000, 6), 2, 8, 150., 203.), ((10, 1000, 1000), 2, 1, 33., 44.)]


@pytest.mark.parametrize("dims,mode,R,tc,fp32", TIMED)
def test_default_takes_the_faster_kernel(cd, dev, dims, mode, R, tc, fp32):
    assert cd.mttkrp_path(dims, mode, R) == ("tensor-core" if tc < fp32 else "cuda-core")
    assert cd.mttkrp_path(dims, mode, R, cd.PREC_BF16X3) == "tensor-core"


@pytest.mark.parametrize("dims", [(37, 8, 8), (7, 200, 200), (3, 5, 7)])
def test_default_is_fp32_where_the_tensor_cores_do_not_apply(cd, dev, dims):
    assert cd.mttkrp_path(dims, 0, 8) == "cuda-core"

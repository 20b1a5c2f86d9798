"""The z pass with a column in registers (planes larger than shared memory):
every transform length it takes and its neighbours, data that end on and off a
lane's last element, mirrored and full tensors, FP32 and FP64.  Tolerances as in
test_gpu_anylength.py, whose comparison with the oracle's lattice sum this uses."""
import pytest

from test_gpu_anylength import _compare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import maglua_b200 as M
    M.init(0)
    return M


@pytest.mark.parametrize("dims", [(4, 512, 9), (4, 256, 32), (3, 128, 33), (2, 64, 65), (2, 64, 128), (2, 32, 129)])
def test_fp32(M, dims):
    _compare(M, dims, "f32", trunc=4)


@pytest.mark.parametrize("dims", [(3, 256, 12), (3, 128, 20), (2, 64, 64)])
def test_fp64(M, dims):
    _compare(M, dims, "f64", trunc=4)


@pytest.mark.parametrize("dims,precision", [((3, 256, 17), "f32"), ((2, 64, 70), "f32"), ((3, 512, 5), "f64"),
                                            ((3, 128, 32), "f64")])
def test_full_tensor(M, dims, precision):
    _compare(M, dims, precision, trunc=4, cell=(1, 0, 0, 0.3, 1, 0, 0.2, 0.1, 1))

"""Launch shapes chosen by the class tuner on the row layouts a lattice may have."""
import pytest
import torch

from tests.gpu_util import require_cuda

pytestmark = pytest.mark.gpu
P = 11000


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    require_cuda()


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "fp64"])
@pytest.mark.parametrize("nz,pitch", [(33, False), (3, False), (2, None), (5, None), (32, None),
                                      (33, None), (33, True)])
def test_tuned_class_gives_a_shape_the_lattice_runs(storage, nz, pitch):
    from funlbm_b200 import tune
    from funlbm_b200.lattice import Lattice

    lat = Lattice(19, (6, 5, nz), [P] * 6, 0.7, storage=storage, pitch=pitch)
    lat.init(None)
    nodes, threads = tune.tune_class(lat)
    assert tune.shape_ok(nodes, lat.pz, tune.STORAGE_BITS[storage], nz)
    assert (lat.desc.step_nodes, lat.desc.step_threads) == (nodes, threads)
    lat.step()
    torch.cuda.synchronize()
    assert lat.read_status() == 0

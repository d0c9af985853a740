"""micropp3_kernel_launches counts every kernel of an assembly by element matrices: two per chunk of element layers."""
import pytest

from cases import gpu_config

pytestmark = pytest.mark.gpu


# all layers in one chunk; layers of 75 MB, of which the ring holds two, so that each is a chunk; four layers per chunk
# (layers of 19.9 MB, five in 96 MB) with a remainder
@pytest.mark.parametrize("size,chunks", [((6, 5, 4), 1), ((128, 128, 5), 5), ((60, 72, 9), 3)])
def test_assembly_launches(gpu_lib, size, chunks):
    import micropp_gb300 as mg
    # the constructor with use_A0 and without the linear ctan runs one assembly and nothing else
    g = mg.Micropp(gpu_config(size, use_A0=1, its_with_A0=1, calc_ctan_lin=0))
    assert g.kernel_launches() == 2 * chunks
    g.close()

"""Device memory that the phases of a fit take on their first use."""
import pytest

from gaspacho2_b200 import synth
from gaspacho2_b200.model import GPLVM

pytestmark = pytest.mark.gpu


def test_many_groups_take_no_split_sums():
    """400 groups x 2,000 genes x 68 dense columns: the group sums go straight to their place (435 MB, there since
    the design was loaded), so the split sums' buffer has to hold none of that. What remains: the pair
    products' buffer (337 MB), the gathered pairs (39 MB), the split products (35 MB) and the code."""
    import torch

    ds = synth.make(2, 3, N=4000, G=2000, M=64, Q=5, init=False)
    ds.init.rho[:] = 3.0
    with GPLVM.from_dataset(ds) as m:
        m.set_params(ds.init)
        m.kernel_mats()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        m.glm_init()
        m.irls_sweep(0, 0)
        used = before - torch.cuda.mem_get_info()[0]
    assert used < 600e6, used

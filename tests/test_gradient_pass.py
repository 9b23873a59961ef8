"""The first pass of the Gauss gradient, which leaves out the products with its zero old
gradient: on geometry that is not finite, where they are NaN, and with a result that shares
memory with the field."""
import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from oracle import oracle
from tests.meshes import oracle_mesh
from tests.test_wave_blocks import box_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where,value", [("xf", np.inf), ("xc", np.nan), ("yf", -np.inf),
                                         ("facint", np.inf)])
@pytest.mark.parametrize("nigrad", [1, 2])
def test_first_gradient_pass_on_odd_geometry(where, value, nigrad):
    """A zero old gradient over an infinite offset is a NaN, as in the oracle's loops."""
    m = box_mesh(5, 4, 3)
    getattr(m, where)[7] = value
    phi = fcg.uniform(5, 2, m.numTotal)
    c = fcg.Context(m)
    with np.errstate(all="ignore"):
        exp = oracle.grad_gauss(oracle_mesh(m), phi, nigrad=nigrad)
    got = c.grad(phi, "gauss", nigrad=nigrad)
    assert np.isnan(exp).any() and np.array_equal(got, exp, equal_nan=True)
    c.close()


@pytest.mark.parametrize("nigrad", [1, 3])
def test_gradient_over_its_own_field(nigrad):
    """phi at the head of the array that takes the result (device memory)."""
    import torch

    m = box_mesh(9, 6, 4)
    c = fcg.Context(m)
    phi = fcg.uniform(5, 2, m.numTotal)
    buf = torch.zeros(max(3 * m.numCells, m.numTotal), dtype=torch.float64, device="cuda")
    buf[:m.numTotal] = torch.from_numpy(phi).cuda()
    torch.cuda.synchronize()
    c._check(c.lib.fcg_grad(c.h, buf.data_ptr(), buf.data_ptr(), 1, nigrad), "fcg_grad")
    torch.cuda.synchronize()
    got = buf[:3 * m.numCells].cpu().numpy().reshape(-1, 3)
    assert np.array_equal(got, oracle.grad_gauss(oracle_mesh(m), phi, nigrad=nigrad))
    c.close()

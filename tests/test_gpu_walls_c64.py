"""One-CTA complex64 walls of every length, in packed FP32 pairs and scalar
(csrc/qsg_evolve1d_inst.cuh says which), against the oracle's wall path.  The bar
is the complex64 path's own, relative L2 <= 1e-5 over these steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 128, 256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("order", [2, 4])
def test_wall_of_every_length_vs_oracle(oracle, n, order):
    import qusim_gb300 as q
    rng = np.random.default_rng(n)
    psi = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    psi[0] = 0
    V = rng.uniform(-1, 1, n)
    ref = oracle.evolve1d(psi, V, 0.1, 0.01, 10, order=order, wall=True)
    inst = q.Instance.create_1d(q.Context(0), psi, V, 0.1, 0.01, order=order, precision="mixed",
                                boundary=q.BoundaryCondition.InfiniteWall)
    inst.step(10)
    got = inst.get_psi()
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)

"""Edges of the fixed-point passes on grids and volumes (csrc/qsg_fix.cuh,
csrc/qsg_evolve3d.cuh): states far from 1 in magnitude, sites and potentials that
are not finite, neighbouring columns of very different size; and the longest
columns of the complex128 Born pass (csrc/qsg_born_inst.cuh).  The bar is the
path's own, relative L2 <= 1e-12 against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.fixture(scope="module")
def qsg():
    import qusim_gb300 as q
    q.load()
    return q


@pytest.fixture(scope="module")
def ctx(qsg):
    return qsg.Context(0)


def rel_l2(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def noise(shape, seed=0):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape), rng.uniform(-1, 1, shape)


def create(qsg, ctx, psi, V, order):
    if psi.ndim == 2:
        return qsg.Instance.create_2d(ctx, psi, V, 0.1, 0.1, 0.01, order=order)
    return qsg.Instance.create_3d(ctx, psi, V, 0.1, 0.1, 0.1, 0.01, order=order)


def reference(oracle, psi, V, steps, order):
    if psi.ndim == 2:
        return oracle.evolve2d(psi, V, 0.1, 0.1, 0.01, steps, order=order)
    return oracle.evolve3d(psi, V, 0.1, 0.1, 0.1, 0.01, steps, order=order)


# 2D: four and eight elements a thread, unsplit columns of 4096, Bluestein; 3D: lines within a warp, of
# several warps and the longest, along each axis
SHAPES = [(128, 128), (512, 256), (4096, 128), (45, 100), (16, 16, 16), (32, 128, 64), (1024, 16, 16),
          (16, 1024, 16), (16, 16, 1024)]
IDS = ["x".join(map(str, s)) for s in SHAPES]


@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
@pytest.mark.parametrize("order", [2, 4])
def test_states_of_any_scale_vs_oracle(qsg, ctx, oracle, shape, order):
    psi, V = noise(shape)
    ref = reference(oracle, psi, V, 2, order)
    # powers of two are exact; near 2^-1000 the smallest components are subnormal (2^-1074 against 2^-1000)
    for k in (0, -1000, -400, 900):
        inst = create(qsg, ctx, np.ldexp(psi.view(np.float64), k).view(np.complex128), V, order)
        inst.step(2)
        got = np.ldexp(inst.get_psi().view(np.float64), -k).view(np.complex128)
        inst.close()
        assert rel_l2(got, ref) <= TOL, k


@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
@pytest.mark.parametrize("bad", [np.inf, np.nan, "V"])
def test_what_is_not_finite_spreads_everywhere(qsg, ctx, shape, bad):
    psi, V = noise(shape)
    site = tuple(n // 3 for n in shape)
    if bad == "V":
        V[site] = np.inf
    else:
        psi[site] = bad
    inst = create(qsg, ctx, psi, V, 4)
    inst.step(1)
    got = inst.get_psi()
    inst.close()
    assert not np.isfinite(got).any()


@pytest.mark.parametrize("shape", SHAPES, ids=IDS)
def test_zero_state_stays_zero(qsg, ctx, shape):
    _, V = noise(shape)
    inst = create(qsg, ctx, np.zeros(shape, np.complex128), V, 4)
    inst.step(3)
    got = inst.get_psi()
    inst.close()
    assert np.all(got == 0)


@pytest.mark.parametrize("shape", [s for s in SHAPES if len(s) == 3], ids=IDS[4:])
@pytest.mark.parametrize("steps", [1, 2, 5])
def test_neighbours_of_very_different_size_3d(qsg, ctx, oracle, shape, steps):
    psi, V = noise(shape, 1)
    for axis, (rate, period) in enumerate(((40.0, 7), (30.0, 5), (20.0, 3))):
        s = np.exp(-rate * (np.arange(shape[axis]) % period))
        psi = psi * s.reshape([-1 if a == axis else 1 for a in range(3)])
    ref = reference(oracle, psi, V, steps, 4)
    inst = create(qsg, ctx, psi, V, 4)
    inst.step(steps)
    got = inst.get_psi()
    inst.close()
    assert rel_l2(got, ref) <= TOL


# complex128 Born columns of 2048 rows (512 threads) and of 4096 (1024 threads): only rows of 4096 leave the
# grid so little split
@pytest.mark.parametrize("nx", [2048, 4096])
def test_born_longest_columns_vs_oracle(qsg, oracle, nx):
    from tests.workloads import born_potential_2d
    ny, hx, hy = 4096, nx / 16, 256.0
    V, _, _ = born_potential_2d(nx, ny, -hx, hx, -hy, hy)
    ref = oracle.born2d(V, -hx, hx, -hy, hy, 2.0, 0.0, dirx=1.0, diry=0.5, order=1, preconditional=True,
                        preconditioner=1, slow=1.0, computes=2)
    per = qsg.QuPerturbation2D()
    opts = qsg.Options().Gb300().Order(1).Slow(1.0).Precision("fp64").Preconditional(True)
    opts.SetString("preconditioner", "Vellekoop")
    per.init(V, -hx, hx, nx, -hy, hy, ny, 2.0, 0.0, 1.0, 0.5, qsg.SolverMethod.BornSerise, 1.0, 1.0, opts)
    per.Compute()
    per.Compute()
    assert rel_l2(per.GetPsi(), ref["dpsi"]) <= TOL

"""The tables that a complex128 Bluestein instance holds: one form of each (fixed
point with a real time step, doubles with a complex one), read by the stepping
kernels and by the kinetic energy alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def qsg():
    import qusim_gb300 as q
    q.load()
    return q


@pytest.fixture(scope="module")
def ctx(qsg):
    return qsg.Context(0)


def create(qsg, ctx, shape, dt, order, wall=False):
    rng = np.random.default_rng(7)
    psi = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    V = rng.uniform(-1, 1, shape)
    if len(shape) == 1:
        bc = qsg.BoundaryCondition.InfiniteWall if wall else qsg.BoundaryCondition.Period
        return qsg.Instance.create_1d(ctx, psi, V, 0.1, dt, order=order, boundary=bc)
    return qsg.Instance.create_2d(ctx, psi, V, 0.1, 0.2, dt, order=order)


# one CTA of every length M = 256 .. 8192, walls, grids with one or both sides Bluestein
SHAPES = [((3,), 0), ((130,), 0), ((500,), 0), ((1000,), 0), ((2000,), 0), ((4095,), 0), ((100,), 1), ((2047,), 1),
          ((45, 100), 0), ((100, 128), 0), ((700, 30), 0), ((3, 2049), 0)]


@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("shape,wall", SHAPES)
def test_real_step_holds_no_second_form(qsg, ctx, shape, wall, order):
    held = {}
    for dt in (0.01, 0.01 - 0.001j, 0.01, 0.01 - 0.001j):  # the second time the context's own tables are there
        before = ctx.bytes_in_use()
        inst = create(qsg, ctx, shape, dt, order, wall)
        held[dt] = ctx.bytes_in_use() - before
        inst.close()
    # a fixed-point potential table ends in a flag entry of 16 bytes
    assert held[0.01] <= held[0.01 - 0.001j] + 16 * (1 if order == 2 else 2)


# Both forms hold the same factors, doubles to 2^-53; a transform's error is a few times that (three
# convolution products and 13 stages at most), and the energy is a ratio of sums of its squares: 1e-14 with
# headroom of ten
@pytest.mark.parametrize("shape,wall", SHAPES)
def test_kinetic_energy_of_both_forms(qsg, ctx, shape, wall):
    a, b = (create(qsg, ctx, shape, dt, 2, wall) for dt in (0.01, 0.01 - 0.001j))
    ka, kb = a.energies()[0], b.energies()[0]
    a.close()
    b.close()
    assert abs(ka - kb) <= 1e-13 * abs(kb)

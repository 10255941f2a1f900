"""The fixed-point line transforms of the complex128 path (csrc/qsg_fix.cuh) at
the edges of their scaling: lines far from 1 in magnitude, impulses and
constants (the extremes of peak against norm), zero and non-finite lines,
neighbouring columns of very different size.  The bar is the path's own,
relative L2 <= 1e-12 against the oracle."""
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


def line(n, kind, seed=0):
    rng = np.random.default_rng(seed)
    if kind == "impulse":
        psi = np.zeros(n, np.complex128)
        psi[n // 3] = 1.0 - 0.5j
    elif kind == "constant":
        psi = np.full(n, 0.75 + 0.25j)
    else:
        psi = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    V = rng.uniform(-1, 1, n)
    return psi, V


# 64: lines of 8 threads; 256: one warp; 512: two warps; 4096: the longest; 1000, 3000: Bluestein;
# 8192, 32768: four-step
@pytest.mark.parametrize("n", [64, 256, 512, 4096, 1000, 3000, 8192, 32768])
@pytest.mark.parametrize("kind", ["impulse", "constant", "noise"])
def test_lines_of_any_scale_vs_oracle(qsg, ctx, oracle, n, kind):
    psi, V = line(n, kind)
    ref = oracle.evolve1d(psi, V, 0.1, 0.01, 3, order=4)
    # powers of two are exact, so the scaled state's result is the scaled result; near 2^-1000 the
    # smallest components are subnormal (2^-1074 against 2^-1000)
    for k in (0, -1000, -400, 900):
        inst = qsg.Instance.create_1d(ctx, np.ldexp(psi.view(np.float64), k).view(np.complex128), V, 0.1, 0.01,
                                      order=4)
        inst.step(3)
        got = np.ldexp(inst.get_psi().view(np.float64), -k).view(np.complex128)
        assert rel_l2(got, ref) <= TOL, k
        inst.close()


@pytest.mark.parametrize("n", [64, 4096, 1000, 8192])
def test_zero_line_stays_zero(qsg, ctx, n):
    _, V = line(n, "noise")
    inst = qsg.Instance.create_1d(ctx, np.zeros(n, np.complex128), V, 0.1, 0.01, order=2)
    inst.step(2)
    assert np.all(inst.get_psi() == 0)


@pytest.mark.parametrize("n", [64, 4096, 8192])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_non_finite_site_spreads_over_the_line(qsg, ctx, n, bad):
    psi, V = line(n, "noise")
    psi[n // 5] = bad
    inst = qsg.Instance.create_1d(ctx, psi, V, 0.1, 0.01, order=2)
    inst.step(1)
    assert not np.isfinite(inst.get_psi()).any()


@pytest.mark.parametrize("shape", [(128, 128), (256, 1024), (4096, 128), (100, 45)])
def test_columns_of_very_different_size_vs_oracle(qsg, ctx, oracle, shape):
    nx, ny = shape
    rng = np.random.default_rng(1)
    psi = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * np.exp(-40.0 * (np.arange(ny) % 7))[None, :]
    psi *= np.exp(-30.0 * (np.arange(nx) % 5))[:, None]
    V = rng.uniform(-1, 1, shape)
    ref = oracle.evolve2d(psi, V, 0.1, 0.1, 0.01, 2, order=4)
    inst = qsg.Instance.create_2d(ctx, psi, V, 0.1, 0.1, 0.01, order=4)
    inst.step(2)
    assert rel_l2(inst.get_psi(), ref) <= TOL


# one CTA, Bluestein, four-step, Bluestein on the four-step passes; walls
@pytest.mark.parametrize("n,wall", [(64, 0), (4096, 0), (1000, 0), (16384, 0), (6000, 0), (512, 1), (700, 1), (4096, 1)])
def test_infinite_potential_gives_nan(qsg, ctx, n, wall):
    psi, V = line(n, "noise")
    V[n // 2] = np.inf
    inst = qsg.Instance.create_1d(ctx, psi, V, 0.1, 0.01, order=4,
                                  boundary=qsg.BoundaryCondition.InfiniteWall if wall else qsg.BoundaryCondition.Period)
    inst.step(1)
    got = inst.get_psi()
    assert not np.isfinite(got[1:]).any()


@pytest.mark.parametrize("shape", [(128, 128), (512, 256), (30, 45)])
def test_infinite_potential_gives_nan_2d(qsg, ctx, shape):
    rng = np.random.default_rng(2)
    psi = rng.standard_normal(shape) + 0j
    V = rng.uniform(-1, 1, shape)
    V[3, 5] = np.inf
    inst = qsg.Instance.create_2d(ctx, psi, V, 0.1, 0.1, 0.01, order=2)
    inst.step(1)
    assert not np.isfinite(inst.get_psi()).any()


@pytest.mark.parametrize("n", [256, 16384])
def test_batch_of_real_and_complex_steps_equals_solo(qsg, ctx, n):
    # real time steps run in fixed point, complex ones in double: two classes of one length
    psis, Vs = zip(*(line(n, "noise", seed) for seed in range(4)))
    dts = [0.01, 0.01 - 0.002j, 0.02, -0.005j]
    b = qsg.Batch(ctx, psis, Vs, [0.1] * 4, dts, order=2)
    if n > 4096:
        plan = next(p for p in qsg.candidate_plans_1d("fp64", n) if p.kind == 1 and p.n1 != b.plan(n).n1)
        b.set_plan(n, plan)
    b.step(5)
    for i in range(4):
        solo = qsg.Instance.create_1d(ctx, psis[i], Vs[i], 0.1, dts[i], order=2)
        if n > 4096:
            solo.set_plan(plan)
        solo.step(5)
        assert np.array_equal(b.instance(i).get_psi(), solo.get_psi()), i


@pytest.mark.parametrize("shape", [(128, 128), (1024, 256), (4096, 128), (256, 512)])
def test_every_2d_plan_vs_oracle(qsg, ctx, oracle, shape):
    # four and eight elements a thread, units of fewer threads, unsplit columns up to 4096, both
    # with fixed-point products (real steps) and double ones (complex steps)
    nx, ny = shape
    rng = np.random.default_rng(4)
    psi = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    V = rng.uniform(-1, 1, shape)
    for dt in (0.01, 0.01 - 0.0005j):
        ref = oracle.evolve2d(psi, V, 0.1, 0.1, dt, 1, order=2)
        inst = qsg.Instance.create_2d(ctx, psi, V, 0.1, 0.1, dt, order=2)
        for plan in inst.candidate_plans():
            inst.set_psi(psi)
            inst.set_plan(plan)
            inst.step(1)
            got = inst.get_psi()
            assert rel_l2(got, ref) <= TOL, (dt, plan.g, plan.row_e, plan.row_nt, plan.col_e, plan.col_w)


# complex128 steps with a real dt: split calls, and reads in between, leave the state as one call does
# (Bluestein lines on the four-step passes apply other table values at a call's ends and agree to rounding)
@pytest.mark.parametrize("n,wall", [(64, 0), (4096, 0), (1000, 0), (300, 0), (16384, 0), (512, 1), (700, 1), (8192, 1)])
@pytest.mark.parametrize("order", [2, 4])
def test_split_calls_equal_one_call(qsg, ctx, n, wall, order):
    psi, V = line(n, "noise")
    bc = qsg.BoundaryCondition.InfiniteWall if wall else qsg.BoundaryCondition.Period
    a = qsg.Instance.create_1d(ctx, psi, V, 0.1, 0.01, order=order, boundary=bc)
    b = qsg.Instance.create_1d(ctx, psi, V, 0.1, 0.01, order=order, boundary=bc)
    a.step(7)
    for k in (3, 1, 3):
        b.step(k)
        b.get_psi()
    assert np.array_equal(a.get_psi(), b.get_psi())


@pytest.mark.parametrize("shape", [(128, 128), (1024, 256), (4096, 128), (45, 100), (100, 128)])
@pytest.mark.parametrize("order", [2, 4])
def test_split_calls_equal_one_call_2d(qsg, ctx, shape, order):
    rng = np.random.default_rng(3)
    psi = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    V = rng.uniform(-1, 1, shape)
    a = qsg.Instance.create_2d(ctx, psi, V, 0.1, 0.1, 0.01, order=order)
    b = qsg.Instance.create_2d(ctx, psi, V, 0.1, 0.1, 0.01, order=order)
    a.step(4)
    for k in (1, 2, 1):
        b.step(k)
        b.get_psi()
    assert np.array_equal(a.get_psi(), b.get_psi())

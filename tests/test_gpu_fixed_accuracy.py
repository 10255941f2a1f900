"""Rounding of the complex128 fixed-point path (csrc/qsg_fix.cuh) against extended
precision: the error of a few steps, and that no rounding has a preferred
direction.

Bounds, from the arithmetic.  A product is off by 0.31 units rms of its result
(uniform rounding, and the part of the low words' product left out), and the unit
is at most 2^-55 of the line's largest component; so is a stage's.  Phase factors
are doubles: a component near 1 is rounded by 3.2e-17 rms, the same at every
application of a table.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EVENT = 0.31 * 2.0 ** -55
FACTOR = 3.2e-17
PEAK = 4.5  # largest component of a line of normal deviates over their rms


@pytest.fixture(scope="module")
def qsg():
    import qusim_gb300 as q
    q.load()
    return q


@pytest.fixture(scope="module")
def ctx(qsg):
    return qsg.Context(0)


def make(qsg, ctx, psi, V, dt, order, wall=False):
    if psi.ndim == 1:
        bc = qsg.BoundaryCondition.InfiniteWall if wall else qsg.BoundaryCondition.Period
        return qsg.Instance.create_1d(ctx, psi, V, 1.0, dt, order=order, boundary=bc)
    if psi.ndim == 2:
        return qsg.Instance.create_2d(ctx, psi, V, 1.0, 1.0, dt, order=order)
    return qsg.Instance.create_3d(ctx, psi, V, 1.0, 1.0, 1.0, dt, order=order)


def evolve_ld(psi, V, dt, steps, wall):
    """O4 steps in long double (hbar = m = 1, spacing 1, double pi and coefficients as the engine has them)."""
    ld = np.longdouble
    t = 2.0 ** (1.0 / 3.0)
    vc = [1 / (2 * (2 - t)), (1 - t) / (2 * (2 - t)), (1 - t) / (2 * (2 - t)), 1 / (2 * (2 - t))]
    tc = [1 / (2 - t), -t / (2 - t), 1 / (2 - t)]
    psi, V = psi.astype(np.clongdouble), V.astype(ld)
    n0 = psi.shape[0]
    dims = [2 * n0] if wall else psi.shape
    k2 = ld(0)
    for a, n in enumerate(dims):
        i = np.arange(n).astype(ld)
        f = np.where(i > n // 2, n - i, i) ** 2 * (2 * ld(math.pi) / n) ** 2 / 2
        k2 = k2 + f.reshape([n if b == a else 1 for b in range(len(dims))])

    def cis(c, x):
        p = ld(c) * ld(dt) * x
        return np.cos(p) - 1j * np.sin(p)

    for _ in range(steps):
        for j, c in enumerate(tc):
            psi = psi * cis(vc[j], V)
            p = psi
            if wall:
                p = np.concatenate([psi, psi[:1] * 0, -psi[1:][::-1]])
                p[0] = 0
            f = np.fft.fftn(p)
            assert f.dtype == np.clongdouble
            psi = np.fft.ifftn(f * cis(c, k2))
            if wall:
                psi = psi[:n0].copy()
                psi[0] = 0
        psi = psi * cis(vc[3], V)
    return psi


# transforms of one kinetic substep and the stages of each: one CTA, Bluestein (two transforms of M for
# one), four-step (two passes and two twiddle products), walls; 2D and 3D per axis
CASES = [((64,), 0, 2, 2), ((256,), 0, 2, 3), ((4096,), 0, 2, 4), ((1000,), 0, 4, 4), ((3000,), 0, 4, 5),
         ((16384,), 0, 2, 10), ((6000,), 0, 4, 10), ((512,), 1, 2, 4), ((700,), 1, 4, 4), ((8192,), 1, 2, 10),
         ((256, 128), 0, 4, 4), ((128, 1024), 0, 4, 4), ((45, 100), 0, 8, 4), ((16, 32, 64), 0, 6, 3)]


@pytest.mark.parametrize("shape,wall,transforms,stages", CASES,
                         ids=["x".join(map(str, c[0])) + ("wall" if c[1] else "") for c in CASES])
def test_error_against_extended_precision(qsg, ctx, shape, wall, transforms, stages):
    rng = np.random.default_rng(11)
    psi = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    V = rng.uniform(-1, 1, shape)
    if wall:
        psi[0] = 0
    steps, dt = 3, 0.01
    inst = make(qsg, ctx, psi, V, dt, 4, wall)
    inst.step(steps)
    got = inst.get_psi()
    inst.close()
    ref = evolve_ld(psi, V, dt, steps, wall)
    err = float(np.sqrt(np.sum(np.abs(got - ref) ** 2) / np.sum(np.abs(ref) ** 2)))
    # per substep: the transforms' stages, a product after each transform and one taking up of the line
    events = 3 * steps * (transforms * (stages + 2))
    # tables: V c1 and c2 twice a step; per axis K d1 twice and K d2 once
    tables = (2 * steps) ** 2 * 2 + len(shape) * ((2 * steps) ** 2 + steps ** 2)
    bound = math.hypot(math.sqrt(events) * EVENT * PEAK, math.sqrt(tables) * FACTOR)
    print(f"{shape} error {err:.3g} bound {bound:.3g}")
    assert err <= 2 * bound


# The sum over the sites is the state's k = 0 amplitude.  With every factor 1 it stays, but for roundings,
# whose errors add like their square root where no direction is preferred: each site's within 0.31 units of
# at most 2^-55 of the largest value (the 1 at one site).  All other sites hold positive values of up to 16
# units, so a direction shows as a shift of all of them.
@pytest.mark.parametrize("n,steps,events,seeds", [(1000, 1, 30, 1), (3000, 1, 30, 1), (4096, 64, 12, 8),
                                                  (16384, 64, 18, 8)])
def test_roundings_prefer_no_direction(qsg, ctx, n, steps, events, seeds):
    shift = np.zeros(2)
    for seed in range(seeds):
        rng = np.random.default_rng(5 + seed)
        psi = (rng.random(n) + (1j * rng.random(n) if seeds > 1 else 0)) * 2.0 ** -54
        psi = psi.astype(np.complex128)
        psi[0] = 1.0
        inst = make(qsg, ctx, psi, np.zeros(n), 1e-30, 2)
        inst.step(steps)
        got = inst.get_psi()
        inst.close()
        shift += [math.fsum(got.real) - math.fsum(psi.real), math.fsum(got.imag) - math.fsum(psi.imag)]
    sigma = math.sqrt(n * events * steps / seeds) * EVENT
    print(f"n {n}: shift {shift / seeds / 2.0 ** -58} of {4 * sigma / 2.0 ** -58:.0f} units")
    assert np.all(np.abs(shift / seeds) <= 4 * sigma)

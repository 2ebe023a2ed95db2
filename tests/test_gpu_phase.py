"""Nonlinear phases on both sides of the evaluations' limits (2^-8 and 1/32)
within one tile: in real time a cell's phase factor follows from its own
argument, so however the tile is cut (row walks, register patches, several steps
per launch, a batch) it carries the same bits.  The double rotating frame is not
among the cases: there a warp chooses one evaluation for all its cells."""
import numpy as np
import pytest

import oracle as O
from helpers import desc_from_params, seeded_case

pytestmark = pytest.mark.gpu

DT, G = 1e-3, 250.0  # g dt |psi|^2 up to 0.08


def _case(N, Ny, per=(False, False), omega=0.0, lhy=0.0, precision=1):
    lat, psi0, V = seeded_case(N, 10.0, Ny, per, omega)
    phase = G * DT * np.abs(psi0) ** 2
    assert phase.min() < 2.0 ** -8 and phase.max() > 1.0 / 32
    assert ((phase > 2.0 ** -8) & (phase < 1.0 / 32)).any()
    p = lat.params(DT, False, 1.0, G, lhy, omega)
    return desc_from_params(p, precision), psi0, O.exp_table(V, DT, False)


def _kernel(desc, psi0, table):
    from trottersuzuki_b200 import Kernel
    k = Kernel(desc)
    k.set_state(psi0)
    k.set_exp_potential(*table)
    return k


@pytest.mark.parametrize("N,Ny", [(97, 61), (301, 304), (850, 401)])
@pytest.mark.parametrize("lhy", [0.0, 0.3])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_steps_taken_together_or_one_by_one(N, Ny, lhy, precision):
    desc, psi0, table = _case(N, Ny, lhy=lhy, precision=precision)
    out = []
    for single in (False, True):
        with _kernel(desc, psi0, table) as k:
            for n in (6, 50):
                if single:
                    for _ in range(n):
                        k.step(exchange=False)
                else:
                    k.evolve(n)
            out.append(k.get_state())
    assert np.isfinite(out[0]).all()
    assert np.array_equal(*out)


@pytest.mark.parametrize("N,Ny,per,omega,precision", [
    (97, 61, (False, False), 0.0, 0), (97, 61, (False, False), 0.0, 1),
    (64, 47, (True, True), 0.0, 1), (70, 61, (True, True), 0.6, 1),
    (345, 341, (True, True), 0.6, 1), (351, 350, (False, False), 0.6, 1)])
def test_patches_and_walks(N, Ny, per, omega, precision):
    desc, psi0, table = _case(N, Ny, per, omega, precision=precision)
    out = []
    for walk in (None, 2, 0):
        with _kernel(desc, psi0, table) as k:
            if walk is not None:
                k.set_walk(walk)
            assert k.launch_shape()["walk"] == (3 if walk is None else walk)
            k.evolve(3)
            k.evolve(40)
            out.append(k.get_state())
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1])
    assert np.array_equal(out[0], out[2])


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_a_pair(precision):
    from trottersuzuki_b200 import Pair
    desc, a0, table = _case(130, 97, precision=precision)
    out = []
    for walk in (None, 2, 0):
        with _kernel(desc, a0, table) as a, _kernel(desc, np.roll(a0, 3, axis=1), table) as b:
            if walk is not None:
                a.set_walk(walk)
                b.set_walk(walk)
            with Pair(a, b, 40.0, 5.0, 2.0, DT) as pair:
                pair.evolve(9)
            out.append((a.get_state(), b.get_state()))
    for x, y in ((0, 1), (0, 2)):
        for i in (0, 1):
            assert np.array_equal(out[x][i], out[y][i])


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_a_batch(precision):
    from trottersuzuki_b200 import Batch
    cases = [_case(97, 61, precision=precision), _case(130, 145, precision=precision)]
    single, batch = ([_kernel(*c) for c in cases] for _ in range(2))
    with Batch(batch) as b:
        b.evolve(40)
        b.synchronize()
    for k, l in zip(single, batch):
        k.evolve(40)
        assert np.array_equal(k.get_state(), l.get_state())
        k.close()
        l.close()

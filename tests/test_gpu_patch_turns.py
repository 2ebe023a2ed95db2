"""Register patches with more regions than blocks resident on 148 SMs (444 blocks
of 2 x 2 patches in double and 592 in float, 296 and 444 of 4 x 4, 296 of the adjoint
pass): a block then takes regions in turn, inner and edge ones, through the same
exchange buffers.  Against the row walks: bits in real time, 1e-13 in imaginary time
(the order of the norm's sum)."""
import numpy as np
import pytest

import oracle as O
from helpers import desc_from_params, seeded_case

pytestmark = pytest.mark.gpu


def _compare(desc, psi0, table, imag, side, places, steps=(3, 37)):
    """The default and the checked walk, past one replayed graph."""
    from trottersuzuki_b200 import Kernel
    out = []
    for walk in (None, 0):
        with Kernel(desc) as k:
            if walk is None:
                shape = k.launch_shape()
                assert (shape["walk"], shape["cells_per_lane"], shape["steps"]) == (3, side, 1)
                assert shape["strips"] * shape["segments"] > places
            else:
                k.set_walk(walk)
            k.set_state(psi0)
            k.set_exp_potential(*table)
            for n in steps:
                k.evolve(n)
            out.append(k.get_state())
    assert np.isfinite(out[0]).all()
    if not imag:
        assert np.array_equal(*out)
    else:
        # float: a last-bit difference of the factor, rounded per step
        bar = 1e-13 if desc.precision == 0 else sum(steps) * 2.0 ** -23
        assert np.abs(out[0] - out[1]).max() <= bar * np.abs(out[1]).max()


# N, Ny, periodic, omega, imaginary time, precision, patch side, resident blocks
@pytest.mark.parametrize("N,Ny,per,omega,imag,precision,side,places", [
    (601, 577, True, 0.0, False, 0, 2, 444), (601, 577, True, 0.0, True, 0, 2, 444),
    (601, 577, False, 0.0, True, 0, 2, 444), (641, 577, True, 0.0, False, 1, 2, 592),
    (641, 577, True, 0.0, True, 1, 2, 592), (1011, 1007, True, 0.0, True, 1, 4, 296),
    (901, 877, True, 0.6, False, 0, 4, 296), (903, 877, False, 0.6, True, 0, 4, 296),
    (1101, 1077, True, 0.6, False, 1, 4, 444), (1101, 1079, True, 0.6, True, 1, 4, 444)])
def test_regions_in_turn(N, Ny, per, omega, imag, precision, side, places):
    # cells 0.16 wide where rounding must not grow (imaginary time: dt / (4 dx^2) = 0.01)
    lat, psi0, V = seeded_case(N, 0.16 * N if imag else 20.0, Ny, (per, per), omega)
    n0 = O.expectations(lat, psi0)["norm2"] if imag else 0.0
    p = lat.params(1e-3, imag, 1.0, 3.0, 0.2, omega, norm0=n0)
    _compare(desc_from_params(p, precision), psi0, O.exp_table(V, 1e-3, imag), imag, side, places)


@pytest.mark.parametrize("N,Ny,precision,places", [(950, 830, 0, 296), (1101, 1077, 1, 444)])
@pytest.mark.parametrize("imag", [False, True], ids=["real", "imag"])
def test_regions_of_a_cylinder_in_turn(N, Ny, precision, places, imag):
    lat = O.Lattice(N, 0.16 * N, Ny, 0.16 * Ny, False, False, cylindrical=True)
    X, Y = lat.coordinates()
    rng = np.random.default_rng(5)
    psi0 = np.exp(-((X - 2.0) ** 2 + Y ** 2) / 300.0) * (1 + 0.05 * rng.uniform(-1, 1, lat.shape))
    psi0 = psi0 * np.exp(0.3j * Y)
    V = 0.005 * (X ** 2 + Y ** 2) + lat.azimuthal(1)
    n0 = O.expectations(lat, psi0)["norm2"] if imag else 0.0
    p = lat.params(1e-3, imag, 1.0, 3.0, 0.0, 0.0, norm0=n0, angular_momentum=1)
    _compare(desc_from_params(p, precision), psi0, O.exp_table(V, 1e-3, imag), imag, 4, places)


def test_regions_of_a_pair_in_turn():
    from trottersuzuki_b200 import Kernel, Pair
    lat, a0, V = seeded_case(601, 20.0, 577, (True, True))
    b0 = np.roll(a0, 3, axis=1)
    table = O.exp_table(V, 1e-3, False)
    out = []
    for walk in (None, 0):
        pa, pb = lat.params(1e-3, False, 1.0, 3.0), lat.params(1e-3, False, 1.2, 2.0)
        with Kernel(desc_from_params(pa)) as a, Kernel(desc_from_params(pb)) as b:
            for k, psi in ((a, a0), (b, b0)):
                if walk is not None:
                    k.set_walk(walk)
                k.set_state(psi)
                k.set_exp_potential(*table)
            with Pair(a, b, 4.0, 5.0, 2.0, 1e-3) as pair:
                shape = a.launch_shape()
                assert shape["walk"] == (3 if walk is None else 0)
                assert walk == 0 or shape["strips"] * shape["segments"] > 444
                pair.evolve(11)
            out.append((a.get_state(), b.get_state()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


def test_regions_with_potential_rows_in_turn():
    import torch
    from trottersuzuki_b200 import Kernel
    lat, psi0, V = seeded_case(601, 20.0, 577)
    p = lat.params(1e-3, False, 1.0, 3.0, 0.2)
    stack = torch.stack([torch.tensor(V * (1 + 0.1 * i), device="cuda") for i in range(3)])
    torch.cuda.synchronize()
    out = []
    for walk in (None, 0):
        with Kernel(desc_from_params(p)) as k:
            if walk is not None:
                k.set_walk(walk)
            k.set_state(psi0)
            k.set_exp_potential(*O.exp_table(V, 1e-3, False))
            # 601 columns: the steps read the rows of an even pitch
            rows = torch.zeros((3, 577, 602), dtype=torch.float64, device="cuda")
            rows[:, :, :601] = stack
            torch.cuda.synchronize()
            k.evolve_potentials(rows.data_ptr(), 602, rows.stride(0), 3, 1e-3)
            out.append(k.get_state())
    assert np.array_equal(*out)


@pytest.mark.parametrize("g,lhy,every,imag", [(0.0, 0.0, 0, False), (8.0, 0.0, 4, False),
                                              (8.0, 0.5, 3, False), (8.0, 0.5, 4, True)])
def test_regions_of_the_adjoint_in_turn(g, lhy, every, imag):
    """431 x 449 is 18 x 19 = 342 regions."""
    import torch
    from trottersuzuki_b200.adjoint import AdjointEngine
    lat, psi0, V = seeded_case(431, 20.0, 449)
    n0 = O.expectations(lat, psi0)["norm2"] if imag else 0.0
    p = lat.params(1e-3, imag, 1.0, g, lhy, norm0=n0)
    v, psi = torch.tensor(V, device="cuda"), torch.tensor(psi0, device="cuda")
    lam = torch.randn(psi.shape, dtype=torch.complex128, device="cuda",
                      generator=torch.Generator("cuda").manual_seed(3))
    out = []
    for rows in (0, 6):
        e = AdjointEngine(desc_from_params(p), 1e-3, 10, every)
        if rows:
            e.set_segments(adjoint_rows=rows)
        e.forward(v, psi)
        out.append([t.cpu().numpy() for t in e.backward(lam)])
        e.close()
    for got, old in zip(*out):
        if imag:
            assert np.abs(got - old).max() <= 1e-13 * np.abs(old).max()
        else:
            assert np.array_equal(got, old)

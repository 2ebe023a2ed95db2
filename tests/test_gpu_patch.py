"""The register-patch step against the checked walk and the oracle.

The patches perform the same operations per cell as the row walks (the same
pair forms, potential row and fused multiply-adds), so in real time a tile
stepped by them carries the checked walk's bits; in imaginary time the squared
norm is summed over another grid of blocks, so the renormalisation factor may
differ in its last bits (1e-13).  The oracle bar is the parity bar, 1e-10.
Sizes lie at the edges of the regions (24 or 56 written cells, 16 or 48 with 8
halo columns) and on either side of the limits between patch sizes.
"""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from helpers import desc_from_params, seeded_case

pytestmark = pytest.mark.gpu

# name, N, Ny, periodic, g, lhy, omega, imag, precision, patch side (cells 10/N
# wide; in float imaginary time 0.16, where dt / (4 dx^2) = 0.01: at 1.8, as 853
# columns over 10 would have it, eight sweeps of cosh(1.8) lose all of float)
CASES = [
    ("one_cell", 1, 1, (False, False), 1.0, 0.0, 0.0, False, 0, 2),
    ("one_row", 50, 1, (False, False), 1.0, 0.0, 0.0, False, 0, 2),
    ("one_column", 1, 50, (False, False), 0.0, 0.0, 0.0, True, 0, 2),
    ("region", 24, 24, (False, False), 5.0, 0.3, 0.0, False, 0, 2),
    ("region_plus_1", 25, 49, (False, False), 5.0, 0.0, 0.0, True, 0, 2),
    ("rim_left", 27, 75, (False, False), 2.0, 0.0, 0.0, False, 0, 2),
    ("interior", 130, 101, (False, False), 2.0, 0.0, 0.0, True, 0, 2),
    ("interior_fp32", 131, 100, (False, False), 2.0, 0.1, 0.0, False, 1, 2),
    ("linear_fp32", 77, 60, (False, False), 0.0, 0.0, 0.0, True, 1, 2),
    ("wide_fp32", 850, 801, (False, False), 2.0, 0.0, 0.0, False, 1, 4),
    ("wide_imag_fp32_coarse", 853, 802, (False, False), 2.0, 0.0, 0.0, True, 1, 4),
    ("periodic", 64, 40, (True, True), 2.0, 0.0, 0.0, False, 0, 2),
    ("periodic_odd", 63, 45, (True, True), 1.0, 0.0, 0.0, False, 0, 2),
    ("periodic_odd_fp32", 63, 45, (True, True), 1.0, 0.0, 0.0, False, 1, 2),
    ("periodic_x", 61, 30, (True, False), 1.0, 0.0, 0.0, True, 0, 2),
    ("periodic_y", 30, 61, (False, True), 1.0, 0.0, 0.0, False, 0, 2),
    ("halo_only", 4, 4, (True, True), 1.0, 0.0, 0.0, False, 0, 2),
    ("rotating", 48, 33, (False, False), 3.0, 0.0, 0.6, False, 0, 2),
    ("rotating_periodic", 70, 61, (True, True), 3.0, 0.0, 0.6, True, 0, 2),
    ("rotating_wide", 345, 341, (True, True), 3.0, 0.2, 0.6, False, 0, 4),
    ("rotating_wide_closed", 351, 350, (False, False), 0.0, 0.0, 0.6, False, 0, 4),
    ("rotating_wide_fp32", 345, 341, (True, True), 3.0, 0.0, 0.6, False, 1, 4),
]


def _close(got, old, imag):
    if imag:
        assert np.abs(got - old).max() <= 1e-13 * np.abs(old).max()
    else:
        assert np.array_equal(got, old)


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_patches_match_checked_walk_and_oracle(case):
    """40 steps in two evolve calls: plain launches and a replayed graph."""
    from trottersuzuki_b200 import Kernel
    _, N, Ny, per, g, lhy, omega, imag, prec, side = case
    length = 0.16 * N if imag and prec else (10.0 if N > 4 else 1.0)
    lat, psi0, V = seeded_case(N, length, Ny, per, omega)
    n0 = O.expectations(lat, psi0)["norm2"] if imag else 0.0
    p = lat.params(1e-3, imag, 1.0, g, lhy, omega, norm0=n0)
    tr, ti = O.exp_table(V, 1e-3, imag)
    out = {}
    for walk in (None, 0):
        with Kernel(desc_from_params(p, prec)) as k:
            if walk is not None:
                k.set_walk(walk)
            else:
                shape = k.launch_shape()
                assert shape["walk"] == 3 and shape["cells_per_lane"] == side
            k.set_state(psi0)
            k.set_exp_potential(tr, ti)
            k.evolve(3)
            k.evolve(37)
            out[walk] = k.get_state()
    if prec == 0:
        _close(out[None], out[0], imag)
        ref = O.evolve(p, O.evolve(p, psi0, tr, ti, 3), tr, ti, 37)
        assert np.abs(out[None] - ref).max() <= 1e-10
    elif not imag:
        assert np.array_equal(out[None], out[0])
    else:
        # a last-bit difference of the factor, rounded to float per step
        assert np.abs(out[None] - out[0]).max() <= 40 * 2.0 ** -23 * np.abs(out[0]).max()


@pytest.mark.parametrize("imag", [False, True], ids=["real", "imag"])
@pytest.mark.parametrize("N,Ny,py,side", [(40, 37, False, 2), (47, 49, True, 2),
                                          (270, 261, False, 2), (330, 310, False, 4)])
def test_patches_on_cylinders(N, Ny, py, side, imag):
    from trottersuzuki_b200 import Kernel
    lat = O.Lattice(N, 8.0, Ny, 10.0, False, py, cylindrical=True)
    X, Y = lat.coordinates()
    rng = np.random.default_rng(5)
    psi0 = np.exp(-((X - 2.0) ** 2 + Y ** 2) / 3.0) * (1 + 0.05 * rng.uniform(-1, 1, lat.shape))
    psi0 = psi0 * np.exp(0.3j * Y)
    V = 0.5 * (X ** 2 + Y ** 2) + lat.azimuthal(1)
    n0 = O.expectations(lat, psi0)["norm2"] if imag else 0.0
    p = lat.params(1e-3, imag, 1.0, 25.0, 0.0, 0.0, norm0=n0, angular_momentum=1)
    tr, ti = O.exp_table(V, 1e-3, imag)
    ref = O.evolve(p, O.evolve(p, psi0, tr, ti, 6), tr, ti, 36)
    out = {}
    for walk in (None, 0):
        with Kernel(desc_from_params(p)) as k:
            if walk is not None:
                k.set_walk(walk)
            else:
                shape = k.launch_shape()
                assert shape["walk"] == 3 and shape["cells_per_lane"] == side
            k.set_state(psi0)
            k.set_exp_potential(tr, ti)
            k.evolve(6)
            k.evolve(36)
            out[walk] = k.get_state()
    assert np.abs(out[None] - ref).max() <= 1e-10 * np.abs(ref).max()
    _close(out[None], out[0], imag)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("N,per,omega", [(40, (False, False), (5.0, 2.0)),
                                         (57, (True, True), (0.0, 0.0)),
                                         (430, (False, False), (5.0, 2.0))])
def test_patches_of_a_pair(N, per, omega, prec):
    """Two species with and without a Rabi coupling: the checked walk's bits
    (430: 324 regions of 2 x 2 patches, 64 of 4 x 4)."""
    from trottersuzuki_b200 import Kernel, Pair
    lat, a0, V = seeded_case(N, 10.0, None, per)
    b0 = np.roll(a0, 3, axis=1)
    tr, ti = O.exp_table(V, 1e-3, False)
    out = {}
    for walk in (None, 0):
        pa, pb = lat.params(1e-3, False, 1.0, 3.0), lat.params(1e-3, False, 1.2, 2.0)
        with Kernel(desc_from_params(pa, prec)) as a, Kernel(desc_from_params(pb, prec)) as b:
            for k, psi in ((a, a0), (b, b0)):
                if walk is not None:
                    k.set_walk(walk)
                k.set_state(psi)
                k.set_exp_potential(tr, ti)
            with Pair(a, b, 4.0, omega[0], omega[1], 1e-3) as pair:
                assert a.launch_shape()["walk"] == (3 if walk is None else 0)
                pair.rabi(0.5)
                pair.evolve(7)
                pair.evolve(4)
            out[walk] = (a.get_state(), b.get_state())
    assert np.array_equal(out[None][0], out[0][0])
    assert np.array_equal(out[None][1], out[0][1])


@pytest.mark.parametrize("W,H", [(24, 24), (26, 51), (130, 100)])
@pytest.mark.parametrize("pad", [0, 2])
def test_patches_with_potential_rows(W, H, pad):
    """Steps that read the potential (rows of any even pitch): the bits of a
    table per step on the checked walk."""
    import torch
    from trottersuzuki_b200 import Kernel
    lat, psi0, V = seeded_case(W, 10.0, H)
    p = lat.params(1e-3, False, 1.0, 3.0, 0.2)
    tr, ti = O.exp_table(V, 1e-3, False)
    stack = torch.zeros((5, H, W + pad), dtype=torch.float64, device="cuda")
    for i in range(5):
        stack[i, :, :W] = torch.tensor(V * (1 + 0.1 * i))
    torch.cuda.synchronize()
    out = {}
    for walk in (None, 0):
        with Kernel(desc_from_params(p)) as k:
            if walk is not None:
                k.set_walk(walk)
            k.set_state(psi0)
            k.set_exp_potential(tr, ti)
            k.evolve_potentials(stack.data_ptr(), W + pad, stack.stride(0), 5, 1e-3)
            k.evolve(2)
            out[walk] = k.get_state()
    assert np.array_equal(out[None], out[0])


# sizes with 8 or 16 written cells per region (3 or 2 steps of 2 x 2 patches), on
# either side of the limit between them, and with 48 (2 steps of 4 x 4)
@pytest.mark.parametrize("N,Ny,precision", [
    (1, 1, 0), (8, 8, 0), (9, 17, 1), (41, 30, 0), (97, 97, 0), (112, 113, 1), (256, 255, 0),
    (301, 304, 0), (391, 390, 1), (501, 530, 0), (770, 815, 0), (1150, 1201, 1)])
@pytest.mark.parametrize("g,lhy", [(0.0, 0.0), (2.0, 0.0), (2.0, 0.3)])
def test_several_steps_per_launch_match_single_steps(N, Ny, precision, g, lhy):
    """evolve() of odd and even numbers of steps, from either buffer, plain and
    replayed: the bits of as many single steps."""
    from trottersuzuki_b200 import Kernel
    lat, psi0, V = seeded_case(N, 0.05 * N, Ny)
    desc = desc_from_params(lat.params(1e-3, False, 1.0, g, lhy), precision=precision)
    pot = np.exp(-1e-3j * V)
    out = []
    for single in (False, True):
        k = Kernel(desc)
        k.set_state(psi0)
        k.set_exp_potential(pot.real.copy(), pot.imag.copy())
        for n in (1, 2, 3, 4, 5, 50, 99):
            if single:
                for _ in range(n):
                    k.step(exchange=False)
            else:
                k.evolve(n)
        out.append(k.get_state())
        k.close()
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("N,Ny", [(1, 1), (24, 24), (25, 49), (131, 90)])
@pytest.mark.parametrize("g,lhy,every,imag", [(0.0, 0.0, 0, False), (8.0, 0.0, 4, False),
                                              (8.0, 0.5, 3, False), (0.0, 0.0, 5, True),
                                              (8.0, 0.5, 4, True)])
def test_adjoint_patches_match_the_row_walk(N, Ny, g, lhy, every, imag):
    """Gradients of 10 steps: the row walk's bits in real time; in imaginary
    time the inner products are summed over another grid of blocks."""
    import torch
    from trottersuzuki_b200.adjoint import AdjointEngine
    lat, psi0, V = seeded_case(N, 10.0 if N > 1 else 1.0, Ny)
    n0 = O.expectations(lat, psi0)["norm2"] if imag else 0.0
    p = lat.params(1e-3, imag, 1.0, g, lhy, norm0=n0)
    v = torch.tensor(V, device="cuda")
    psi = torch.tensor(psi0, device="cuda")
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
        _close(got, old, imag)


@pytest.mark.parametrize("W,H,pad,shift", [(1, 1, 0, 0), (5, 3, 2, 0), (1023, 2, 1, 1),
                                           (1025, 7, 0, 0), (2050, 3, 3, 1), (31, 300, 0, 1)])
@pytest.mark.parametrize("precision,imag", [(0, False), (0, True), (1, False), (1, True)])
def test_device_state_and_table_copies(W, H, pad, shift, precision, imag):
    """States and tables from and to device rows of any pitch; shift: rows that
    start half an element off its alignment (states in real time only go in)."""
    import torch
    from trottersuzuki_b200 import Kernel
    lat, psi0, V = seeded_case(W, 0.2 * W, H)
    p = lat.params(1e-3, imag, 1.0, 1.0, 0.0, norm0=1.0 if imag else 0.0)
    real = torch.float32 if precision else torch.float64
    ctype = torch.complex64 if precision else torch.complex128
    k = Kernel(desc_from_params(p, precision=precision))

    def rows(a, n):  # n reals per element, `shift` reals into an allocation
        flat = torch.zeros(H * (W + pad) * n + shift, dtype=real, device="cuda")
        r = flat[shift:].view(H, W + pad, n)
        r[:, :W] = a
        return r

    src = torch.tensor(psi0, device="cuda").to(ctype)
    r = rows(torch.view_as_real(src), 2)
    k.set_state_device(r.data_ptr(), W + pad)
    out = torch.full((H, W + pad), 7.0, dtype=ctype, device="cuda")
    k.get_state_device(out.data_ptr(), W + pad)
    assert torch.equal(out[:, :W], src)
    assert bool((out[:, W:] == 7).all())
    k.close()
    # the table: the same step as with whole rows side by side
    tab = torch.tensor(np.exp((-1e-3 if imag else -1e-3j) * V), device="cuda")
    tab = tab.to(real)[..., None] if imag else torch.view_as_real(tab.to(ctype))
    n = tab.shape[-1]
    steps = []
    for r, pitch in ((rows(tab, n), W + pad), (tab.contiguous(), W)):
        with Kernel(desc_from_params(p, precision=precision)) as k:
            k.set_state_device(src.data_ptr(), W)
            k.set_exp_potential_device(r.data_ptr(), pitch)
            k.step(exchange=False)
            steps.append(k.get_state())
    assert np.array_equal(*steps, equal_nan=True)


def test_asking_for_a_walk_or_overlap_after_steps_keeps_the_evolution():
    """Switches of walk and launch mode between evolve calls that replay graphs."""
    from trottersuzuki_b200 import Kernel
    from trottersuzuki_b200._capi import lib
    lat, psi0, V = seeded_case(100, 10.0, 90, (True, True))
    p = lat.params(1e-3, False, 1.0, 2.0)
    tr, ti = O.exp_table(V, 1e-3, False)
    res = []
    for switch in (False, True):
        with Kernel(desc_from_params(p)) as k:
            k.set_state(psi0)
            k.set_exp_potential(tr, ti)
            k.evolve(70)
            if switch:
                assert lib().ts_b200_set_overlap(k.handle, C.c_int(1)) == 0
            k.evolve(70)
            if switch:
                k.set_walk(2)
                assert k.launch_shape()["walk"] == 2
            k.evolve(70)
            k.step(True)
            k.step(False)
            res.append(k.get_state())
    assert np.array_equal(res[0], res[1])


# tiles of few rows and many columns: patches while their regions are resident at
# once or few beside what a walk would take, else the walk
@pytest.mark.parametrize("N,Ny,imag,precision,cyl,walk", [
    (50000, 1, False, 0, False, 2), (50000, 9, False, 0, False, 2), (50000, 3, True, 1, False, 2),
    (24000, 1, True, 0, False, 2), (50000, 9, False, 1, True, 2), (5000, 9, False, 0, False, 3),
    (11000, 24, True, 0, False, 3), (1, 20000, False, 0, False, 3)])
def test_wide_tiles_of_few_rows_are_walked(N, Ny, imag, precision, cyl, walk):
    from trottersuzuki_b200 import Kernel
    if cyl:
        lat = O.Lattice(N, 0.2 * N, Ny, 0.2 * Ny, False, False, cylindrical=True)
    else:
        lat = O.Lattice(N, 0.2 * N, Ny, 0.2 * Ny)
    rng = np.random.default_rng(2)
    psi0 = 0.1 * (rng.standard_normal(lat.shape) + 1j * rng.standard_normal(lat.shape))
    V = rng.uniform(0.0, 2.0, lat.shape)
    n0 = O.expectations(lat, psi0)["norm2"] if imag else 0.0
    p = lat.params(1e-3, imag, 1.0, 2.0, 0.0, norm0=n0)
    out = []
    for checked in (False, True):
        with Kernel(desc_from_params(p, precision)) as k:
            if checked:
                k.set_walk(0)
            k.set_state(psi0)
            k.set_exp_potential(*O.exp_table(V, 1e-3, imag))
            k.evolve(5)
            assert k.launch_shape()["walk"] == (0 if checked else walk)
            out.append(k.get_state())
    if imag and precision:
        assert np.abs(out[0] - out[1]).max() <= 5 * 2.0 ** -23 * np.abs(out[1]).max()
    else:
        _close(*out, imag)


@pytest.mark.parametrize("N,Ny,every,imag", [(32000, 1, 0, False), (44000, 3, 4, False),
                                             (44000, 1, 4, True), (16000, 9, 0, False)])
def test_adjoint_of_wide_tiles_of_few_rows(N, Ny, every, imag):
    """The pass on its default (the walk beyond the resident regions where that has
    less to do) and on the walk asked for."""
    import torch
    from trottersuzuki_b200.adjoint import AdjointEngine
    lat = O.Lattice(N, 0.2 * N, Ny, 0.2 * Ny)
    rng = np.random.default_rng(4)
    psi0 = 0.1 * (rng.standard_normal(lat.shape) + 1j * rng.standard_normal(lat.shape))
    n0 = O.expectations(lat, psi0)["norm2"] if imag else 0.0
    p = lat.params(1e-3, imag, 1.0, 8.0 if every else 0.0, norm0=n0)
    v = torch.tensor(rng.uniform(0.0, 2.0, lat.shape), device="cuda")
    psi = torch.tensor(psi0, device="cuda")
    out = []
    for rows in (0, 6):
        e = AdjointEngine(desc_from_params(p), 1e-3, 10, every)
        if rows:
            e.set_segments(adjoint_rows=rows)
        e.forward(v, psi)
        out.append([t.cpu().numpy() for t in e.backward(psi)])
        e.close()
    for got, old in zip(*out):
        _close(got, old, imag)


@pytest.mark.parametrize("precision,imag", [(0, False), (1, True)])
def test_states_and_tables_not_of_this_gpu_are_copied_by_the_runtime(precision, imag):
    """Rows in pinned host memory stand for all memory that the handle's GPU does not
    own: no kernel reads them."""
    import torch
    from trottersuzuki_b200 import Kernel
    from trottersuzuki_b200.kernel import launch_count
    lat, psi0, V = seeded_case(45, 10.0, 31)
    p = lat.params(1e-3, imag, 1.0, 1.0, 0.0, norm0=1.0 if imag else 0.0)
    ctype = torch.complex64 if precision else torch.complex128
    src = torch.tensor(psi0).to(ctype)
    tab = torch.tensor(np.exp((-1e-3 if imag else -1e-3j) * V))
    tab = tab.to(torch.float32 if precision else torch.float64) if imag else tab.to(ctype)
    out = []
    for place in (lambda t: t.pin_memory(), lambda t: t.cuda()):
        with Kernel(desc_from_params(p, precision=precision)) as k:
            s, t = place(src), place(tab)
            before = launch_count()
            k.set_state_device(s.data_ptr(), lat.dim_x)
            k.set_exp_potential_device(t.data_ptr(), lat.dim_x)
            out.append(launch_count() - before)
            k.step(exchange=False)
            out.append(k.get_state())
    assert (out[0], out[2]) == (0, 2)
    assert np.array_equal(out[1], out[3])


def test_device_states_and_tables_under_capture():
    """A stream capture takes the setters, a step and the state's copy."""
    import torch
    from trottersuzuki_b200 import Kernel
    lat, psi0, V = seeded_case(45, 10.0, 31)
    p = lat.params(1e-3, False, 1.0, 1.0)
    src = torch.tensor(psi0, device="cuda")
    tab = torch.tensor(np.exp(-1e-3j * V), device="cuda")
    out = torch.zeros_like(src)
    with Kernel(desc_from_params(p)) as k:
        def program():
            k.set_state_device(src.data_ptr(), lat.dim_x)
            k.set_exp_potential_device(tab.data_ptr(), lat.dim_x)
            k.evolve(3)
            k.get_state_device(out.data_ptr(), lat.dim_x)
        stream = torch.cuda.Stream()
        k.set_stream(stream.cuda_stream)
        with torch.cuda.stream(stream):
            program()
            torch.cuda.synchronize()
            ref = out.clone()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                program()
            out.zero_()
            graph.replay()
            torch.cuda.synchronize()
        assert torch.equal(out, ref)
        k.set_stream(0)


# side of the patches, steps per launch, rows written by a region
@pytest.mark.parametrize("N,per,imag,precision,side,steps,rows", [
    (64, False, False, 0, 2, 3, 8), (200, False, False, 0, 2, 2, 16), (700, False, False, 0, 4, 2, 48),
    (1200, False, False, 1, 4, 2, 48), (64, True, False, 0, 2, 1, 24), (64, False, True, 0, 2, 1, 24)])
def test_launch_shape_tells_what_evolve_launches(N, per, imag, precision, side, steps, rows):
    from trottersuzuki_b200 import Kernel
    from trottersuzuki_b200.kernel import launch_count
    lat, psi0, V = seeded_case(N, 10.0, None, (per, per))
    p = lat.params(1e-4, imag, 1.0, 1.0, 0.0, norm0=1.0 if imag else 0.0)
    with Kernel(desc_from_params(p, precision)) as k:
        k.set_state(psi0)
        k.set_exp_potential(*O.exp_table(V, 1e-4, imag))
        shape = k.launch_shape()
        assert (shape["walk"], shape["cells_per_lane"]) == (3, side)
        assert (shape["steps"], shape["segment_rows"]) == (steps, rows)
        across = -(-lat.dim_x // rows)
        assert (shape["strips"], shape["segments"]) == (across, -(-lat.dim_y // rows))
        before = launch_count()
        k.evolve(6)
        assert launch_count() - before == 6 // steps
        k.set_walk(2)
        assert (k.launch_shape()["walk"], k.launch_shape()["steps"]) == (2, 1)

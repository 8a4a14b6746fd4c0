"""The first solve of a loaded state: its cycles end where they ended before the
solve was two sweeps.

A cycle ends at the first vector with |xi| >= rho, which rounding decides.  In a
channel with wavy walls, whose first solve has ||b'|| set by the few nodes next to
a wall, one vector more or less is percents of omega beside them.  The vectors
built, recorded from the library when it still stored the powers and summed
their Gram matrix in a pass of its own, are therefore part of the result; every
form has to build them, and then agrees in the fields to their rounding."""
import numpy as np
import pytest

from komegafoulingmodel_b200 import Lattice, desc_default
from komegafoulingmodel_b200 import geometry as G

pytestmark = pytest.mark.gpu

# (wave amplitude, vectors of omega, of k) by channel size
RECORDED = {
    (301, 66): [
        (3.0, 3, 4), (3.1, 4, 4), (3.2, 3, 4), (3.3, 4, 4), (3.4, 3, 4), (3.5, 3, 4), (3.6, 3, 5),
        (3.7, 4, 4), (3.8, 4, 6), (3.9, 3, 4), (4.0, 3, 4), (4.1, 4, 5), (4.2, 4, 4), (4.3, 4, 4),
        (4.4, 5, 4), (4.5, 4, 4), (4.6, 4, 5), (4.7, 5, 6), (4.8, 4, 6), (4.9, 4, 5), (5.0, 4, 5),
        (5.1, 4, 4), (5.2, 3, 5), (5.3, 4, 4), (5.4, 5, 5), (5.5, 3, 4), (5.6, 3, 4), (5.7, 3, 4),
        (5.8, 3, 4), (5.9, 3, 4),
    ],
    (640, 130): [
        (6.0, 3, 6), (6.2, 3, 4), (6.4, 3, 6), (6.6, 4, 6), (6.8, 4, 4), (7.0, 3, 7), (7.2, 3, 4),
        (7.4, 4, 4), (7.6, 4, 6), (7.8, 4, 6), (8.0, 3, 6), (8.2, 4, 6), (8.4, 4, 6), (8.6, 4, 4),
        (8.8, 3, 4), (9.0, 3, 4), (9.2, 3, 6), (9.4, 3, 4), (9.6, 3, 4), (9.8, 3, 4), (10.0, 4, 4),
        (10.2, 4, 6), (10.4, 4, 6), (10.6, 4, 4), (10.8, 4, 6),
    ],
}


def _start(nx, ny, amp, nu=5e-4, um=0.05):
    """Walls and a running channel's state: omega of a near wall, k ~ d^2."""
    h = 0.5 * amp * (1 - np.cos(2 * np.pi * np.arange(nx) / nx))
    h = np.round(h * 2.0 ** 20) / 2.0 ** 20  # the same whatever the last digit of the cosine
    yb, yt = 0.5 + h, ny - 1.5 - h
    y = np.arange(ny)[:, None]
    fl = (y > yb) & (y < yt)
    fl[0] = fl[-1] = False
    d = np.where(fl, np.minimum(y - yb, yt - y), 1.0)
    u = np.where(fl, um * 4 * (y - yb) * (yt - y) / (yt - yb) ** 2, 0.0)
    px = [2 / 3 - u * u, 0.5 * (1 / 3 + u + u * u), 0.5 * (1 / 3 - u + u * u)]
    py = [2 / 3, 1 / 6, 1 / 6]
    f = np.stack([px[int(cx)] * py[int(cy)] for cx, cy in zip(G.CX, G.CY)]) * fl
    k = np.where(fl, 1e-5 * (1 - np.exp(-(d / 3) ** 2)), 0.0)
    om = np.where(fl, np.sqrt(1e-6 + (6 * nu / (0.075 * d * d)) ** 2), 0.0)
    s = np.zeros((3, ny, nx))
    s[1] = np.where(fl, 0.5 * um * 4 * (yt + yb - 2 * y) / (yt - yb) ** 2, 0.0)
    nut = np.where(fl, k / np.where(fl, om, 1), 0.0)
    return nu, yb, yt, [np.ascontiguousarray(a).ravel() for a in (f, k, om, nut, s)]


@pytest.mark.parametrize("nx,ny", RECORDED)
def test_cycles_end_as_recorded_in_every_form(kofm_lib, nx, ny):
    wrong = []
    for amp, *vectors in RECORDED[nx, ny]:
        nu, yb, yt, state = _start(nx, ny, amp)
        fields = []
        for form in (0, 2, 3):
            d = desc_default()
            d.nx, d.nx_full, d.ny, d.komega_classic = nx, nx, ny, form
            d.tau, d.fterm, d.mu, d.use_komega = 1.0 / (3 * nu + 0.5), 1e-7, nu, 1
            with Lattice(d) as L:
                L.set_walls(yb, yt)
                for load in range(2):  # whatever the solves of an earlier state took
                    L.set_state(*state)
                    L.step(1)
                    L.sync()
                    st = L.stats()
                    if [st.omega_vectors, st.k_vectors] != vectors:
                        wrong.append((amp, form, load, st.omega_vectors, st.k_vectors, vectors))
                    got = L.get_state()[1:3]
                    if load == 0:
                        fields.append(got)
                        L.step(5)
                    else:
                        assert all(map(np.array_equal, got, fields[-1])), (amp, form)
        # the same coefficients on the same powers: their FP64 sum, in another
        # order, and one rounding to FP32
        for got in fields[1:]:
            for a, b, start in zip(got, fields[0], state[1:3]):
                bound = np.finfo(np.float32).eps * np.abs(b) + 64 * np.finfo(float).eps * np.abs(start).max()
                assert np.all(np.abs(a - b) <= bound), (amp, np.abs(a - b).max())
    assert not wrong, wrong


@pytest.mark.parametrize("amp,omega,powers", [(0.0, None, 0), (0.0, 2e3, 10), (3.0, None, 10)])
def test_states_that_need_the_fixed_order_take_it(kofm_lib, amp, omega, powers):
    """Straight half-way walls need none; a node near a wall, or omega above the wall
    rows' cap anywhere, does.  Seen in the launches: a first solve in the fixed
    order has one per power and one for the sums, where a march has one."""
    nx, ny = 301, 66
    nu, yb, yt, state = _start(nx, ny, amp)
    if omega:
        state[2][(ny // 2) * nx + 7] = omega
    d = desc_default()
    d.nx, d.nx_full, d.ny, d.komega_classic = nx, nx, ny, 3
    d.tau, d.fterm, d.mu, d.use_komega = 1.0 / (3 * nu + 0.5), 1e-7, nu, 1
    with Lattice(d) as L:
        L.set_walls(yb, yt)
        L.set_state(*state)
        L.step(1)
        L.sync()
        st = L.stats()
        assert st.solver_launches == 3 * st.solver_rounds + powers

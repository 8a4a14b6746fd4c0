"""The two-sweep solve at the edges of its strips, rings and level counts: the
correction it leaves in the fields satisfies the assembled rows.

The rows (kofm_debug_komega_rows) are FP64 and so are the fields of the FP64
form, so the residual b' - A d of d = (field after) - (field before) can be
formed on the host.  Bound: the solve stops at ||b' - A d|| <= relTol ||b'||
(checked with b' - A d summed in another order: a factor 1.01), and d carries
the rounding of the fields it was added to, at most eps ||(I + |N|) |field||| <=
2.5 eps ||field|| with the off-diagonals' row sums below 1.5."""
import numpy as np
import pytest

from komegafoulingmodel_b200 import Lattice, _abi, desc_default
from komegafoulingmodel_b200 import geometry as G
from tests.cases import komega_state, perturbed_state

pytestmark = pytest.mark.gpu

REL_TOL = 1.0e-11


def _matvec(coef, x, ny, nx):
    """A x with unit diagonal; coef [4, ny, nx] E, W, N, S; periodic in x."""
    n = np.vstack([x[1:], np.zeros((1, nx))])
    s = np.vstack([np.zeros((1, nx)), x[:-1]])
    return x + coef[0] * np.roll(x, -1, 1) + coef[1] * np.roll(x, 1, 1) + coef[2] * n + coef[3] * s


@pytest.mark.parametrize("form", [0, 2])
@pytest.mark.parametrize("nx,ny,krylov", [
    (4, 5, 10),      # a strip wraps around the channel many times
    (31, 18, 10), (200, 9, 10),           # narrower than a strip: wraps on both sides
    (236, 12, 10), (237, 12, 10),         # one strip of 10 levels exactly, and one column more
    (256, 34, 10), (257, 34, 10),         # one block's columns, and one more
    (480, 21, 8), (481, 21, 8),           # two strips of 8 levels
    (610, 66, 9), (1001, 130, 7),         # not multiples of anything
    (300, 40, 1), (300, 40, 2), (300, 40, 3), (300, 40, 4), (300, 40, 5), (300, 40, 6),
    (2100, 300, 10),                      # several units a block of the one-launch form
])
def test_solved_fields_satisfy_the_rows(kofm_lib, form, nx, ny, krylov):
    ch = G.straight_channel(nx, ny)
    f = perturbed_state(ch, seed=3, u_mean=0.05, rho_amp=1e-4, u_amp=5e-3, neq_amp=1e-5)
    k, o, nut, s = komega_state(ch, seed=4)
    d = desc_default()
    d.nx, d.nx_full, d.ny = nx, nx, ny
    d.tau, d.fterm, d.mu = 1.0 / (3 * 1e-3 + 0.5), 1e-7, 1e-3
    d.use_komega, d.storage = 1, _abi.STORE_FP64
    d.komega_rel_tol, d.komega_abs_tol = REL_TOL, 0.0
    d.krylov_dim, d.komega_classic = krylov, form
    d.komega_max_iters = 10000
    with Lattice(d) as L:
        L.set_geometry(ch.ntype, ch.wallD, ch.dX)
        L.set_state(f, k, o, nut, s)
        L.lb_step()
        for _ in range(2):  # the second solve starts from the first one's cycle lengths
            L.komega_assemble(1.0)
            before = L.get_state()
            rows = [L.komega_rows(i) for i in range(2)]
            status, _, _ = L.komega_solve(raise_on_error=False)
            after = L.get_state()
            assert status == 0
            for (coef, rhs), x0, x1 in zip(rows, (before[2], before[1]), (after[2], after[1])):
                coef, rhs = coef.reshape(4, ny, nx), rhs.reshape(ny, nx)
                x0, x1 = x0.reshape(ny, nx), x1.reshape(ny, nx)
                fl = ch.fluid_mask()
                r = (rhs - _matvec(coef, (x1 - x0) * fl, ny, nx)) * fl
                bound = 1.01 * REL_TOL * np.linalg.norm(rhs) + 2.5 * np.finfo(float).eps * np.linalg.norm(x1)
                assert np.abs(coef).sum(0).max() < 1.5
                assert np.linalg.norm(r) <= bound, (np.linalg.norm(r), bound)


@pytest.mark.parametrize("krylov,storage", [(2, _abi.STORE_FP64), (10, _abi.STORE_FP64), (3, _abi.STORE_FP32)])
def test_restarts_and_substeps_finish_on_the_device(kofm_lib, krylov, storage):
    """Restarts, and the sub-steps after a NaN residual, of the update that is
    enqueued without a host round trip: the fields of the host-driven rounds.
    Each solve's residual is at most REL_TOL ||b'||, which with off-diagonal row
    sums of at most q < 1 moves d by REL_TOL ||b'|| / (1 - q) at any node; four
    solves (the last two of the sub-steps), and a factor 2 for what a difference
    adds to the next rows.  FP32 fields add a rounding a solve."""
    nx, ny = 301, 43
    ch = G.straight_channel(nx, ny)
    f = perturbed_state(ch, seed=3, u_mean=0.05, rho_amp=1e-4, u_amp=5e-3, neq_amp=1e-5)
    k, o, nut, s = komega_state(ch, seed=4)
    got = []
    for form in (0, 3):
        d = desc_default()
        d.nx, d.nx_full, d.ny = nx, nx, ny
        d.tau, d.fterm, d.mu = 1.0 / (3 * 1e-3 + 0.5), 1e-7, 1e-3
        d.use_komega, d.storage = 1, storage
        d.komega_rel_tol, d.komega_abs_tol = REL_TOL, 0.0
        d.krylov_dim, d.komega_classic = krylov, form
        d.komega_max_iters = 10000
        with Lattice(d) as L:
            L.set_geometry(ch.ntype, ch.wallD, ch.dX)
            L.set_state(f, k, o, nut, s)
            L.step(2)
            _, K, O, _, _ = L.get_state()
            st = L.stats()
            assert max(st.omega_restarts, st.k_restarts) > 2  # more than the first cycle
            L.debug_fail_solves(1, mask=1)  # the next solve reports a NaN residual: two sub-steps
            L.step(1)
            st = L.stats()
            assert st.steps_per_lb == 2
            _, K2, O2, _, _ = L.get_state()
            rows = [L.komega_rows(i) for i in (1, 0)]
            got.append((K, O, K2, O2))
    eps = np.finfo(np.float32 if storage == _abi.STORE_FP32 else np.float64).eps
    for i, (a, b) in enumerate(zip(*got)):
        coef, rhs = rows[i % 2]
        q = np.abs(coef.reshape(4, -1)).sum(0).max()
        bound = 4 * 2 * 2 * REL_TOL * np.linalg.norm(rhs) / (1 - q) + 4 * eps * np.abs(a).max()
        assert q < 1 and np.abs(a - b).max() <= bound, (i, q, np.abs(a - b).max(), bound)


@pytest.mark.parametrize("nx,ny,krylov,storage", [
    (300, 43, 2, _abi.STORE_FP64), (96, 26, 3, _abi.STORE_FP64),  # the second: a lattice that stays in L1
    (300, 43, 10, _abi.STORE_FP64), (300, 43, 3, _abi.STORE_FP32),
])
def test_substeps_with_restarts_of_a_wavy_channel_in_one_launch(kofm_lib, nx, ny, krylov, storage):
    """Both systems' residuals reported as NaN once: four sub-steps, three of them
    assembled, solved with restarts and applied by the launch that finishes an
    update, and four more in the step after; against the host-driven rounds, whose
    assemblies and sweeps are launches of their own.  Bound as above, with the
    largest right-hand side met and seven solves."""
    ch = G.wavy_channel(nx, ny, 0.05 * ny, nx // 2)
    f = perturbed_state(ch, seed=5, u_mean=0.05, rho_amp=1e-4, u_amp=5e-3, neq_amp=1e-5)
    k, o, nut, s = komega_state(ch, seed=6)
    got, norms, q = [], [], 0.0
    for form in (0, 3):
        d = desc_default()
        d.nx, d.nx_full, d.ny = nx, nx, ny
        d.tau, d.fterm, d.mu = 1.0 / (3 * 1e-3 + 0.5), 1e-7, 1e-3
        d.use_komega, d.storage = 1, storage
        d.komega_rel_tol, d.komega_abs_tol = REL_TOL, 0.0
        d.krylov_dim, d.komega_classic = krylov, form
        d.komega_max_iters = 10000
        fields = []
        with Lattice(d) as L:
            L.set_geometry(ch.ntype, ch.wallD, ch.dX, ch.ibb_idx, ch.ibb_q)
            L.set_state(f, k, o, nut, s)
            L.step(2)
            for fail in (1, 0):
                if fail:
                    L.debug_fail_solves(1, mask=3)
                L.step(1)
                st = L.stats()
                assert st.steps_per_lb == 4 and max(st.omega_restarts, st.k_restarts) > 2
                _, K, O, _, _ = L.get_state()
                fields += [O, K]
                for i in (0, 1):
                    coef, rhs = L.komega_rows(i)
                    norms.append(np.linalg.norm(rhs))
                    q = max(q, np.abs(coef.reshape(4, -1)).sum(0).max())
        got.append(fields)
    eps = np.finfo(np.float32 if storage == _abi.STORE_FP32 else np.float64).eps
    assert q < 1
    for i, (a, b) in enumerate(zip(*got)):
        rhs = max(norms[i % 2::2])
        bound = 7 * 2 * 2 * REL_TOL * rhs / (1 - q) + 7 * eps * np.abs(a).max()
        assert np.abs(a - b).max() <= bound, (i, q, np.abs(a - b).max(), bound)


@pytest.mark.parametrize("form", [0, 2, 3])
def test_cycles_cut_by_the_diagonal_of_r(kofm_lib, form):
    """A cycle that ends because diag(R) fell below relTol R(0, 0) back-substitutes
    with R indexed by the vectors kept, where from two on it meets entries that no
    vector wrote: they are zero, the update is not finite, and the solve reports a
    NaN residual and leaves the field.  Against the form of one vector per sweep:
    the same outcome, and the same fields but for the rounding of sums of 12,000
    products (sqrt(12000) eps = 2.4e-14).  Here omega keeps one vector, k one at
    0.1 and two at 0.03."""
    nx, ny = 300, 40
    ch = G.straight_channel(nx, ny)
    state = (perturbed_state(ch, seed=3, u_mean=0.05, rho_amp=1e-4, u_amp=5e-3, neq_amp=1e-5),
             *komega_state(ch, seed=4, s_amp=0.1))

    def solves(form, tol):
        d = desc_default()
        d.nx, d.nx_full, d.ny = nx, nx, ny
        d.tau, d.fterm, d.mu = 1.0 / (3 * 1e-3 + 0.5), 1e-7, 1e-3
        d.use_komega, d.storage, d.komega_classic = 1, _abi.STORE_FP64, form
        d.komega_rel_tol, d.komega_abs_tol = tol, 0.0
        with Lattice(d) as L:
            L.set_geometry(ch.ntype, ch.wallD, ch.dX)
            for _ in range(3):  # the later ones meet what the earlier ones left in shared memory
                L.set_state(*state)
                L.lb_step()
                L.komega_assemble(1.0)
                L.komega_solve(raise_on_error=False)
                st = L.stats()
                counts = [(st.omega_iters, st.omega_vectors, st.omega_nan), (st.k_iters, st.k_vectors, st.k_nan)]
                yield counts, L.get_state()[2:0:-1]

    kept = []
    for tol in (0.1, 0.03):
        list(solves(form, 1e-4))  # full cycles: R filled
        counts, fields = next(solves(1, tol))
        kept += [iters for iters, vectors, _ in counts if iters == vectors - 1]  # one test of xi fewer: cut by diag(R)
        for got, got_fields in solves(form, tol):
            assert got == counts, tol
            for a, b in zip(got_fields, fields):
                assert np.abs(a - b).max() <= 1e-13 * np.abs(b).max(), (tol, got)
    assert kept == [1, 1, 1, 2], kept


@pytest.mark.parametrize("nx,ny,krylov,restarts", [(600, 220, 10, 3), (1100, 960, 3, 3), (1100, 960, 1, 5)])
def test_further_rounds_of_an_update(kofm_lib, nx, ny, krylov, restarts):
    """Lattices and tolerances at which the update's second and later cycles are
    launches of their own (2^17 nodes with 8 vectors a cycle and more, 2^20 with
    fewer), with more rounds than those launches (1 vector), fewer (after a step
    that converges sooner), and sub-steps: the host-driven rounds' fields, the
    bound as above with eleven solves."""
    ch = G.straight_channel(nx, ny)
    f = perturbed_state(ch, seed=3, u_mean=0.05, rho_amp=1e-4, u_amp=5e-3, neq_amp=1e-5)
    k, o, nut, s = komega_state(ch, seed=4)
    got, norms, q = [], [], 0.0
    for form in (0, 3):
        d = desc_default()
        d.nx, d.nx_full, d.ny = nx, nx, ny
        d.tau, d.fterm, d.mu = 1.0 / (3 * 1e-3 + 0.5), 1e-7, 1e-3
        d.use_komega, d.storage = 1, _abi.STORE_FP64
        d.komega_rel_tol, d.komega_abs_tol = REL_TOL, 0.0
        d.krylov_dim, d.komega_classic = krylov, form
        d.komega_max_iters = 10000
        fields = []
        with Lattice(d) as L:
            L.set_geometry(ch.ntype, ch.wallD, ch.dX)
            L.set_state(f, k, o, nut, s)
            for fail in (0, 0, 1, 0):
                if fail:
                    L.debug_fail_solves(1, mask=3)
                L.step(1)
                st = L.stats()
                assert max(st.omega_restarts, st.k_restarts) >= restarts
                _, K, O, _, _ = L.get_state()
                fields += [O, K]
                for i in (0, 1):
                    coef, rhs = L.komega_rows(i)
                    norms.append(np.linalg.norm(rhs))
                    q = max(q, np.abs(coef.reshape(4, -1)).sum(0).max())
            assert st.steps_per_lb == 4
        got.append(fields)
    assert q < 1
    for i, (a, b) in enumerate(zip(*got)):
        rhs = max(norms[i % 2::2])
        bound = 11 * 2 * 2 * REL_TOL * rhs / (1 - q) + 11 * np.finfo(float).eps * np.abs(a).max()
        assert np.abs(a - b).max() <= bound, (i, q, np.abs(a - b).max(), bound)

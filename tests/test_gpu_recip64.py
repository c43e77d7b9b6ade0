"""FP64 reciprocal space (k_ksk64, k_sk_reduce64, k_kforce64) against the oracle's
kwald where its integer sums can go wrong: one structure-factor chunk over every
site (carries between the limbs and the pass to FP64 happen inside the kernel),
ragged last chunks, k_max beyond 15 (scaled |kz| weights), charges of any scale.
The bound is the FP64 parity bound of the force tests (1e-9 relative)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# sites: 6, 30, 129 (below a carry: 128), 387 (ragged), 1536 (48 chunks: beyond the 512-site pass)
@pytest.mark.parametrize("N,eps,n_sc,scale", [(2, 1e-6, 1, 1.0), (10, 1e-12, 1, 1.0), (43, 1e-6, 1, 37.0), (129, 1e-9, 1, 1e-3),
                                              (129, 1e-6, 5, 1.0), (512, 1e-6, 1, 1.0), (512, 1e-6, 0, 1.0)])
def test_kwald_matches_the_oracle(gpu_lib, N, eps, n_sc, scale):
    import ctypes as C

    from oracle.binding import Oracle, _d

    q = gpu_lib
    st = q.seeded_start(N, 1, 298.0, seed=N)
    box = st.box_bohr * np.array([1.0, 1.1, 0.95])
    sites = np.ascontiguousarray(st.q)
    o = Oracle(N, 1, box, 298.0, 0.25, eps_ewald=eps)
    s = q.System.create(N, 1, box, precision=q.FP64, propagator=q.TROTTER, eps_ewald=eps)
    s.ctx.set_tuning(n_sc=n_sc)
    charge = np.ascontiguousarray(s.charges() * scale)
    ref, got = np.zeros_like(sites), np.zeros_like(sites)
    e_ref = o.L.qo_kwald(C.byref(o.s), _d(sites), _d(ref), _d(charge), 0)
    e_got = s.kwald(sites, got, charge)
    assert np.linalg.norm(got - ref) < 1e-9 * np.linalg.norm(ref)
    assert abs(e_got - e_ref) < 1e-9 * abs(e_ref)


# 512 sites in phase at k = (8, 0, 0) whose scaled charge is 1, and just below it: their
# products fill 63 bits, in one structure-factor chunk
@pytest.mark.parametrize("top", [1.0, 1.0 - 2.0 ** -35, 0.5])
def test_coherent_sites_at_the_charge_scale(gpu_lib, top):
    import ctypes as C

    from oracle.binding import Oracle, _d

    q = gpu_lib
    N, L = 512, 47.0
    rng = np.random.default_rng(11)
    x = rng.uniform(0.0, L, size=(3 * N, 3))
    x[:512, 0] = L * (np.arange(512) % 8) / 8.0
    sites = np.ascontiguousarray(x.reshape(1, -1))
    charge = np.where(np.arange(3 * N) < 512, top, -0.5 * top)
    o = Oracle(N, 1, np.full(3, L), 298.0, 0.25, eps_ewald=1e-6)
    s = q.System.create(N, 1, np.full(3, L), precision=q.FP64, propagator=q.TROTTER, eps_ewald=1e-6)
    assert s.info.k_max >= 8
    s.ctx.set_tuning(n_sc=1)
    ref, got = np.zeros_like(sites), np.zeros_like(sites)
    e_ref = o.L.qo_kwald(C.byref(o.s), _d(sites), _d(ref), _d(charge), 0)
    e_got = s.kwald(sites, got, charge)
    assert np.linalg.norm(got - ref) < 1e-9 * np.linalg.norm(ref)
    assert abs(e_got - e_ref) < 1e-9 * abs(e_ref)


# cells so long that k_max reaches the kernels' limit: 2 |kz| + 1 vectors a column in a batch of
# 128, and phase rows of k_max + 1 entries in shared memory. Beyond it the cell is refused.
@pytest.mark.parametrize("axis,ratio,kmax", [(2, 7.1, 62), (0, 7.1, 62), (2, 7.5, 65), (0, 7.5, 65)])
def test_long_cells(gpu_lib, axis, ratio, kmax):
    from oracle.binding import Oracle

    q = gpu_lib
    st = q.seeded_start(27, 1, 298.0, seed=4)
    stretch = np.ones(3)
    stretch[axis] = ratio
    box = st.box_bohr * stretch
    x = st.q.reshape(27, 3, 3)
    pos = np.ascontiguousarray((x - x[:, :1] + x[:, :1] * stretch).reshape(1, -1))
    o = Oracle(27, 1, box, 298.0, 0.25, eps_ewald=1e-6)
    point, lst, _ = o.build_lists(pos)
    ref = np.zeros_like(pos)
    e_ref, _ = o.force_eval_trotter(pos, ref, point, lst)
    for prec, tol in ((q.FP64, 1e-9), (q.MIXED, 1e-4)):
        if kmax > 63 and (prec == q.FP64 or axis == 2):
            with pytest.raises(q.QtgError) as ei:
                q.System.create(27, 1, box, precision=prec, propagator=q.TROTTER)
            assert ei.value.status == 1
            continue
        s = q.System.create(27, 1, box, precision=prec, propagator=q.TROTTER)
        assert s.info.k_max == kmax
        got = np.zeros_like(pos)
        e_got, _ = s.force_eval_trotter(pos, got, s.charges(), point, lst)
        assert np.linalg.norm(got - ref) < tol * np.linalg.norm(ref)
        self_e = s.info.kappa / np.sqrt(np.pi) * float((s.charges() ** 2).sum())
        assert abs(e_got - e_ref) < (1e-9 if prec == q.FP64 else 1e-6) * max(abs(e_ref), self_e)

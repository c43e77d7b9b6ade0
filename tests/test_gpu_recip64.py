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

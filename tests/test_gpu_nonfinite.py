"""FP64 evaluations of configurations with a coordinate or charge that is not finite: its
phases make every reciprocal sum NaN, and with them the energy and the forces of every
molecule, as a caller's check of the forces expects. A later evaluation of a sound
configuration by the same context is sound again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BAD = [np.nan, np.inf, -np.inf]


# molecules: one ragged preparation block, and several a dimension; the site in the first, a middle, the last block
@pytest.mark.parametrize("N,P", [(3, 1), (64, 3), (129, 1)])
@pytest.mark.parametrize("bad", BAD)
def test_forces_of_every_molecule(gpu_lib, N, P, bad):
    q = gpu_lib
    st = q.seeded_start(N, P, 298.0, seed=N, density_g_cm3=0.6)
    s = q.System.create(N, P, st.box_bohr, precision=q.FP64, propagator=q.TROTTER)
    good = np.ascontiguousarray(st.q)
    point, lst, _ = s.build_lists(good)
    ref = np.zeros_like(good)
    e_ref, _ = s.force_eval_trotter(good, ref, s.charges(), point, lst)
    for at in (0, 9 * (N // 2) + 4, 9 * N - 1):  # an oxygen's x (its M site), an H's y, the last H's z
        pos, f = good.copy(), np.zeros_like(good)
        pos[P - 1, at] = bad
        s.force_eval_trotter(pos, f, s.charges(), point, lst)
        assert np.all(np.isnan(f[P - 1]))
        assert np.allclose(f[:P - 1], ref[:P - 1], rtol=0, atol=1e-12)  # the other configurations are their own
        f1 = np.zeros_like(good)
        assert np.isnan(s.get_forces_nospline(pos, f1, s.charges(), point, lst, P - 1))
        assert np.all(np.isnan(f1[P - 1]))
    charge = s.charges()
    charge[3 * (N // 2) + 1] = bad
    f = np.zeros_like(good)
    e, _ = s.force_eval_trotter(good, f, charge, point, lst)
    assert np.isnan(e) and np.all(np.isnan(f))
    e, _ = s.force_eval_trotter(good, f, s.charges(), point, lst)
    assert e == pytest.approx(e_ref, rel=1e-12) and np.allclose(f, ref, rtol=0, atol=1e-12)


@pytest.mark.parametrize("bad", BAD)
def test_kwald(gpu_lib, bad):
    q = gpu_lib
    st = q.seeded_start(64, 1, 298.0, seed=3)
    s = q.System.create(64, 1, st.box_bohr, precision=q.FP64, propagator=q.TROTTER)
    sites = np.ascontiguousarray(st.q)
    sites[0, 100] = bad
    f = np.zeros_like(sites)
    assert np.isnan(s.kwald(sites, f, s.charges()))
    assert np.all(np.isnan(f))
    sites[0, 100], charge = 1.0, s.charges()
    charge[7] = bad
    f[:] = 0.0
    assert np.isnan(s.kwald(sites, f, charge))
    assert np.all(np.isnan(f))


@pytest.mark.parametrize("bad", BAD)
def test_kwald_without_allocation(gpu_lib, bad):
    import ctypes as C

    import torch

    q = gpu_lib
    st = q.seeded_start(64, 1, 298.0, seed=3)
    box = np.ascontiguousarray(st.box_bohr)
    for what in ("sites", "charge", "nothing"):
        sites, charge = torch.from_numpy(st.q.reshape(-1).copy()).cuda(), torch.from_numpy(q.default_charges(64)).cuda()
        if what == "sites":
            sites[571] = bad
        if what == "charge":
            charge[100] = bad
        f, e = torch.zeros_like(sites), torch.zeros(1, dtype=torch.float64, device="cuda")
        status = q.load().qtg_kwald_noalloc(C.c_void_p(sites.data_ptr()), C.c_void_p(charge.data_ptr()), 192,
                                            box.ctypes.data_as(C.POINTER(C.c_double)), 1e-6, C.c_void_p(f.data_ptr()),
                                            C.c_void_p(e.data_ptr()), None)
        torch.cuda.synchronize()
        assert status == 0
        if what == "nothing":
            assert bool(torch.isfinite(f).all()) and bool(torch.isfinite(e).all())
        else:
            assert bool(torch.isnan(f).all()) and bool(torch.isnan(e).all())

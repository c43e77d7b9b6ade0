"""Mixed force evaluation of batches large enough for the kernels that fill the GPU
(launch_real_half's two sites a lane and its like), at ragged and even/odd tile
counts and in orthorhombic cells, against the FP64 form of the same batch (itself
pinned to the oracle). The bound is the mixed form's force tolerance, 1e-4 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(q, N, P, n_sys, ratio, prec):
    st = [q.seeded_start(N, P, 298.0, seed=10 * N + k, density_g_cm3=0.7) for k in range(n_sys)]
    box = st[0].box_bohr * np.array([ratio, 1.0, 1.0 / ratio])
    ctx = q.Context([q.system_desc(N, P, box, propagator=q.TROTTER, thermostat=q.PILE_G, seed=k) for k in range(n_sys)], prec)
    for s, t in zip(ctx.systems, st):
        s.set_state(t.q, t.p)
    ctx.init_forces()
    f = np.concatenate([s.get_state()["fphys"] for s in ctx.systems])
    e = np.array([s.estimators()["pot"][-1] for s in ctx.systems])
    ctx.close()
    return f, e


# sites: 12 (one ragged tile), 66, 129, 192 (full tiles), 258, 321, 648
@pytest.mark.parametrize("N,P,n_sys,ratio", [(4, 128, 10, 1.0), (22, 128, 3, 1.0), (43, 128, 2, 1.1), (64, 128, 2, 1.0),
                                             (86, 96, 1, 0.95), (107, 64, 1, 1.0), (216, 32, 1, 1.05)])
def test_mixed_forces_match_fp64(gpu_lib, N, P, n_sys, ratio):
    q = gpu_lib
    f64, e64 = _batch(q, N, P, n_sys, ratio, q.FP64)
    f32, e32 = _batch(q, N, P, n_sys, ratio, q.MIXED)
    assert np.linalg.norm(f32 - f64) < 1e-4 * np.linalg.norm(f64)
    # energies: 1e-6 of the Ewald self-energy of the bead average (the force tests' bound)
    s = q.System.create(N, 1, q.seeded_start(N, 1, 298.0, seed=1, density_g_cm3=0.7).box_bohr)
    self_e = 0.5 * 2.0 * s.info.kappa / np.sqrt(np.pi) * float((s.charges() ** 2).sum())
    assert np.all(np.abs(e32 - e64) < 1e-6 * self_e)

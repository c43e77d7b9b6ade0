"""FP64 real-space Ewald (k_real64) against the oracle at the edges of its tiles,
packing and pair-function table: ragged and even/odd tile counts, orthorhombic
cells, an Ewald tolerance whose pairs leave the table at its upper end, and a
near-contact pair below its lower end. The bound is the FP64 parity bound of the
force tests (1e-9 relative; summation order is the only difference)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forces(q, N, P, box, pos, eps):
    from oracle.binding import Oracle

    o = Oracle(N, P, box, 298.0, 0.25, eps_ewald=eps)
    s = q.System.create(N, P, box, precision=q.FP64, propagator=q.TROTTER, eps_ewald=eps)
    point, lst, _ = o.build_lists(pos)
    ref, got = np.zeros_like(pos), np.zeros_like(pos)
    e_ref, _ = o.force_eval_trotter(pos, ref, point, lst)
    e_got, _ = s.force_eval_trotter(pos, got, s.charges(), point, lst)
    return ref, got, e_ref, e_got


# 3N sites: 6 (one ragged tile), 30/33 (one / two tiles), 63, 66 (two, three), 129 (five), 192 (six, full)
@pytest.mark.parametrize("N,P,eps,ratio", [(2, 1, 1e-6, 1.0), (10, 1, 1e-6, 1.0), (11, 2, 1e-6, 1.2), (21, 1, 1e-6, 1.0),
                                           (22, 3, 1e-4, 0.9), (43, 1, 1e-6, 1.1), (64, 2, 1e-6, 1.0), (27, 1, 3e-15, 1.0)])
def test_forces_match_the_oracle(gpu_lib, N, P, eps, ratio):
    q = gpu_lib
    st = q.seeded_start(N, P, 298.0, seed=N, density_g_cm3=0.6)
    box = st.box_bohr * np.array([ratio, 1.0, 1.0 / ratio])
    pos = np.ascontiguousarray(st.q)
    ref, got, e_ref, e_got = _forces(q, N, P, box, pos, eps)
    assert np.linalg.norm(got - ref) < 1e-9 * np.linalg.norm(ref)
    assert abs(e_got - e_ref) < 1e-9 * max(1.0, abs(e_ref))


def test_near_contact_pair(gpu_lib):
    q = gpu_lib
    st = q.seeded_start(27, 1, 298.0, seed=5)
    pos = np.ascontiguousarray(st.q)
    # an H of molecule 1 beside an H of molecule 0: (kappa r)^2 near 2^-22, below the table
    pos[0, 9 + 3: 9 + 6] = pos[0, 3:6] + np.array([1e-3, 2e-4, -3e-4])
    ref, got, e_ref, e_got = _forces(q, 27, 1, st.box_bohr, pos, 1e-6)
    assert np.linalg.norm(got - ref) < 1e-9 * np.linalg.norm(ref)
    assert abs(e_got - e_ref) < 1e-9 * abs(e_ref)


# Ewald tolerances whose pairs are beyond the fixed-point form (every pair in FP64), and a
# pair in each of its octaves' neighbours: H...H distances around (kappa r)^2 = 2^-3
@pytest.mark.parametrize("eps,gap", [(1e-18, None), (1e-6, 0.98), (1e-6, 1.02)])
def test_edges_of_the_fixed_point_form(gpu_lib, eps, gap):
    q = gpu_lib
    st = q.seeded_start(27, 1, 298.0, seed=6)
    pos = np.ascontiguousarray(st.q)
    if gap is not None:
        kappa = q.System.create(27, 1, st.box_bohr, precision=q.FP64, propagator=q.TROTTER, eps_ewald=eps).info.kappa
        pos[0, 9 + 3: 9 + 6] = pos[0, 3:6] + gap * 2.0 ** -1.5 / kappa * np.array([0.6, 0.0, 0.8])
    ref, got, e_ref, e_got = _forces(q, 27, 1, st.box_bohr, pos, eps)
    assert np.linalg.norm(got - ref) < 1e-9 * np.linalg.norm(ref)
    assert abs(e_got - e_ref) < 1e-9 * max(1.0, abs(e_ref))


# r_c is half the side of boxes of this size: an H of another molecule just inside it along
# one axis, where FP32 cannot tell the nearer image
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("gap", [1e-9, 1e-8, 3e-8])
def test_pair_at_half_a_side(gpu_lib, axis, gap):
    q = gpu_lib
    st = q.seeded_start(8, 1, 298.0, seed=9, density_g_cm3=0.2)
    for k in range(24):
        pos = np.ascontiguousarray(st.q).copy()
        i, j = k % 8, (k + 1 + k // 8) % 8
        x = pos.reshape(8, 3, 3)
        x[j] += x[i, 1] - x[j, 1]
        x[j, :, axis] += (1.0 if k % 2 else -1.0) * (0.5 - gap) * st.box_bohr[axis]
        ref, got, e_ref, e_got = _forces(q, 8, 1, st.box_bohr, pos, 1e-4)
        assert np.linalg.norm(got - ref) < 1e-9 * np.linalg.norm(ref)
        assert abs(e_got - e_ref) < 1e-9 * max(1.0, abs(e_ref))

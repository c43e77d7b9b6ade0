"""Lists built and handed over whole: every bead by one build, and force calls that
take up no more of the caller's list than its rows reach."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(q, n, p, precision, seed):
    st = q.seeded_start(n, p, 298.0, seed=seed, density_g_cm3=0.7)
    s = q.System.create(n, p, st.box_bohr, precision, propagator=q.TROTTER)
    return s, np.ascontiguousarray(st.q)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,p", [(2, 1), (33, 3), (150, 4), (256, 2)])
def test_lists_by_one_build_and_by_reach(gpu_lib, n, p, precision):
    q = gpu_lib
    prec = q.FP64 if precision == "fp64" else q.MIXED
    s, pos = _system(q, n, p, prec, n)
    point, lst, disp = s.new_lists()
    disp[:] = 1.0
    for b in range(p):
        s.neighbour_list(pos, point, lst, disp, b)
    assert np.all(disp == 0.0)
    point1, lst1, disp1 = s.build_lists(pos)
    assert np.array_equal(point, point1) and np.array_equal(lst, lst1) and np.array_equal(disp1, disp)
    charge = s.charges()

    def forces(sys_, pt, ls):
        f = np.zeros_like(pos)
        e = sys_.force_eval_trotter(pos, f, charge, pt, ls)
        g = np.zeros_like(pos)
        eb = [sys_.get_forces_nospline(pos, g, charge, pt, ls, b) for b in range(p)]
        return f, g, np.array([*e, *eb])

    want = forces(s, point, lst)
    # entries that no row reaches are not read, whatever they hold
    cap = s.info.list_size
    junk = lst.copy()
    for b in range(p):
        junk[b * cap + point[b * n + n - 1]:(b + 1) * cap] = -7
    # a call whose rows are all empty leaves a short list behind, the next a full one
    fresh, _ = _system(q, n, p, prec, n)
    forces(fresh, np.zeros_like(point), junk)
    for got in (forces(s, point, junk), forces(fresh, point, lst)):
        for a, b in zip(got, want):
            scale = np.abs(b).max()
            assert np.abs(a - b).max() <= (1e-12 if precision == "fp64" else 2e-6) * scale
    # a row that reaches past the list is refused as before
    if n > 2:
        bad = point.copy()
        bad[n - 1] = cap + 5
        with pytest.raises(RuntimeError):
            s.force_eval_trotter(pos, np.zeros_like(pos), charge, bad, lst)

"""Mixed reciprocal space of beads large enough for k_ksk2, through kwald against the FP64
form: k_max on both sides of the k-force's instances and of k_ksk2's limit, and sites in
phase (ions on a lattice, whose Bragg vectors add every site's charge in one direction).

The bound on a site's force is the sum over the vectors of 2 c |k| |q| (|S| 2^-24 n + |dS|):
n = 24 roundings between S and the force (weights, column factors, phases to two powers, |kz|
sums and the closing products), and dS = 2^-24 (30 sum |q|) for the chains of 16 sites and
six such sums, the halves and blocks they join, the phases and the column factors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bound(x, charge, box, info):
    b, km = 2.0 * np.pi / box, info.k_max
    g = np.stack(np.meshgrid(np.arange(km + 1), np.arange(-km, km + 1), np.arange(-km, km + 1), indexing="ij"), -1).reshape(-1, 3)
    k2 = ((g * b) ** 2).sum(1)
    g = g[(k2 > 0) & (k2 <= info.kc ** 2)]
    k2 = ((g * b) ** 2).sum(1)
    c = 2.0 * np.pi / np.prod(box) * np.exp(-k2 / (4.0 * info.kappa ** 2)) / k2 * np.where(g[:, 0] > 0, 2.0, 1.0)
    rows = [np.exp(2j * np.pi * np.outer(np.arange(-km, km + 1), x[:, d] / box[d])) for d in range(3)]
    s = np.empty(len(g), complex)
    for kx in range(km + 1):  # by columns: S(k) = sum q X Y Z
        on = g[:, 0] == kx
        for ky in np.unique(g[on, 1]):
            at = on & (g[:, 1] == ky)
            s[at] = rows[2][g[at, 2] + km] @ (charge * rows[0][kx + km] * rows[1][ky + km])
    u = 2.0 ** -24
    return np.abs(charge).max() * float((2.0 * c * np.sqrt(k2) * u * (24.0 * np.abs(s) + 30.0 * np.abs(charge).sum())).sum())


@pytest.mark.parametrize("N,ratio,kind", [(2048, 1.0, "water"), (2304, 1.0, "salt"), (2304, 1.0, "like"), (2048, 1.5, "water"),
                                          (2048, 2.0, "like"), (2048, 2.3, "water")])
def test_kwald_matches_fp64(gpu_lib, N, ratio, kind):
    q = gpu_lib
    st = q.seeded_start(N, 1, 298.0, seed=N)
    box = st.box_bohr * np.array([ratio ** -0.5, ratio ** -0.5, ratio])
    n, rng = 3 * N, np.random.default_rng(N)
    if kind == "water":
        x, charge = st.q.reshape(n, 3) * (box / st.box_bohr), q.default_charges(N)
    else:
        side = (16, 24, 18) if N == 2304 else (16, 16, 24)
        g = np.stack(np.meshgrid(*[np.arange(a) for a in side], indexing="ij"), -1).reshape(-1, 3)
        x = (g + 0.3) * (box / np.array(side)) + rng.normal(scale=0.01, size=(n, 3))
        charge = np.where(g.sum(1) % 2, -1.0, 1.0) if kind == "salt" else np.full(n, 0.7)
    # what both forms can hold: FP32 charges, coordinates in units of 2^-32 of the box
    charge = charge.astype(np.float32).astype(np.float64)
    sites = np.ascontiguousarray((np.round(x / box * 2.0 ** 32) / 2.0 ** 32 * box).reshape(1, -1))
    got = {}
    for prec in (q.FP64, q.MIXED):
        s = q.System.create(N, 1, box, precision=prec, propagator=q.TROTTER)
        f = np.zeros_like(sites)
        got[prec] = s.kwald(sites, f, charge), f
        info = s.info
        s.ctx.close()
    bound = _bound(sites.reshape(n, 3), charge, box, info)
    assert np.abs(got[q.MIXED][1] - got[q.FP64][1]).max() < bound
    assert abs(got[q.MIXED][0] - got[q.FP64][0]) < 1e-4 * abs(got[q.FP64][0])

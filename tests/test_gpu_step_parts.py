"""Steps of many systems taken in parts on their own streams, against the same systems
stepped alone: states and records after NVE steps (no random numbers, whose counters
name the system), and thermostatted steps that stay finite and record every step. The
bound on the momenta is the mixed form's force tolerance, 1e-4 of the impulse."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
STEPS = 3


# two, three and many parts; uneven systems, one of which is most of the work; below the limit
@pytest.mark.parametrize("sizes", [[(512, 32), (512, 32)], [(343, 32), (216, 32), (512, 32), (125, 16)],
                                   [(64, 8)] * 40 + [(512, 24)] + [(128, 32)] * 3, [(216, 8)] * 4])
def test_parts_match_systems_alone(gpu_lib, sizes):
    q = gpu_lib
    st = [q.seeded_start(n, p, 298.0, seed=k, density_g_cm3=0.9) for k, (n, p) in enumerate(sizes)]
    kw = dict(propagator=q.TROTTER, thermostat=q.PILE_G)
    ctx = q.Context([q.system_desc(n, p, s.box_bohr, seed=k, **kw) for k, ((n, p), s) in enumerate(zip(sizes, st))], q.MIXED)
    for s, t in zip(ctx.systems, st):
        s.set_state(t.q, t.p)
    ctx.init_forces()
    ctx.run_steps(STEPS, is_nvt=False)
    ctx.sync()
    dt = 0.25 * 41.341374575751
    for k in sorted({0, 1, len(sizes) // 2, len(sizes) - 1}):
        n, p = sizes[k]
        alone = q.Context([q.system_desc(n, p, st[k].box_bohr, seed=k, **kw)], q.MIXED)
        alone.systems[0].set_state(st[k].q, st[k].p)
        alone.init_forces()
        alone.run_steps(STEPS, is_nvt=False)
        want, got = alone.systems[0].get_state(), ctx.systems[k].get_state()
        impulse = STEPS * dt * np.linalg.norm(want["f"])
        assert np.linalg.norm(got["fphys"] - want["fphys"]) <= 1e-4 * np.linalg.norm(want["fphys"])
        assert np.linalg.norm(got["p"] - want["p"]) <= 1e-4 * impulse
        a, b = ctx.systems[k].estimators(), alone.systems[0].estimators()
        for name in b:
            assert len(a[name]) == len(b[name])
        assert np.allclose(a["pot"], b["pot"], rtol=0, atol=1e-4 * max(1.0, abs(b["pot"][0])))
        alone.close()
    before = len(ctx.systems[0].estimators()["pot"])
    ctx.run_steps(50, is_nvt=True)
    ctx.sync()
    for s in ctx.systems:
        e = s.estimators()
        assert len(e["pot"]) == before + 50
        assert all(np.all(np.isfinite(v)) for v in e.values())
    ctx.close()


# NVT: the parts draw the centroid's random numbers for their own systems and add the ring's
# heat in a range of their own. A last system of the Suzuki-Chin kind, which keeps the step
# in one part, leaves the others' systems, seeds and so random numbers as they are. The bound
# is as above, on the impulse and on the heat, whose terms are the kinetic energy's size.
@pytest.mark.parametrize("sizes,thermostat", [([(343, 32), (216, 32), (512, 32), (125, 32)], "PILE_G"), ([(512, 32)] * 2, "PILE_L"),
                                              ([(216, 8)] * 4, "PILE_G")])
def test_thermostatted_parts_match_one(gpu_lib, sizes, thermostat):
    q = gpu_lib
    st = [q.seeded_start(n, p, 298.0, seed=k, density_g_cm3=0.9) for k, (n, p) in enumerate(sizes + [(8, 2)])]
    got, launches = [], []
    for whole in (False, True):
        kinds = [q.TROTTER] * len(sizes) + [q.SUZUKI_CHIN] * whole
        ctx = q.Context([q.system_desc(s.n_mols, s.n_beads, s.box_bohr, seed=k, propagator=kind, thermostat=getattr(q, thermostat))
                         for k, (s, kind) in enumerate(zip(st, kinds))], q.MIXED)
        for s, t in zip(ctx.systems, st):
            s.set_state(t.q, t.p)
        ctx.init_forces()
        ctx.sync()
        before = ctx.kernel_launches()
        ctx.run_steps(STEPS, is_nvt=True)
        ctx.sync()
        launches.append((ctx.kernel_launches() - before) // STEPS)
        got.append([(s.get_state(), s.estimators()) for s in ctx.systems[:len(sizes)]])
        ctx.close()
    split = sum(n * p for n, p in sizes) >= 32000
    assert (launches[0] > 20) == split  # a part's launches are some ten, a whole step's fourteen
    dt = 0.25 * 41.341374575751
    for (a, ea), (b, eb), (n, p) in zip(*got, sizes):
        assert np.linalg.norm(a["p"] - b["p"]) <= 1e-4 * STEPS * dt * np.linalg.norm(b["f"])
        assert len(ea["pot"]) == len(eb["pot"])
        assert np.allclose(ea["heat"], eb["heat"], rtol=0, atol=1e-4 * eb["kin"][0])
        assert np.allclose(ea["kin"], eb["kin"], rtol=1e-4)
        assert np.allclose(ea["pot"], eb["pot"], rtol=0, atol=1e-4 * max(1.0, abs(eb["pot"][0])))

"""Which steps of a trajectory rebuild the lists, and who decides it: no list period at all, replica
groups, and lists outrun in one group only.  The same schedule gives the same bits; other schedules
are held against one call per step."""
import numpy as np
import pytest

from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import MOIL_NB_FP64, MOIL_NB_MIXED, Nonbonded

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def waters(n, seed, speed):
    """A water box with rigid translations of the given spread (Å/ps)."""
    s = S.water_box(n, 18.62 if n == 216 else (n / S.WATER_DENSITY) ** (1 / 3), seed)
    rng = np.random.Generator(np.random.PCG64(seed))
    return s, np.repeat(rng.normal(0.0, speed, (n, 3)), 3, axis=0)


def start(systems):
    x = torch.tensor(np.concatenate([s.coor for s, _ in systems]), device="cuda")
    v = torch.tensor(np.concatenate([v for _, v in systems]), device="cuda")
    m = torch.tensor(np.tile([15.9994, 1.008, 1.008], x.shape[0] // 3), device="cuda")
    torch.cuda.synchronize()
    return x, v, m


def run(nb, state, steps, dt=0.0005, calls=1):
    x, v, m = state[0].clone(), state[1].clone(), state[2]
    torch.cuda.synchronize()
    for _ in range(calls):
        es, ek = nb.md_step(x.data_ptr(), v.data_ptr(), m.data_ptr(), dt, steps)
    return x, v, [e["e_total"] for e in es], ek


def test_negative_list_period_is_none():
    """A period of -1 means no period, as 0 does: rebuilds wherever a site has moved half the skin."""
    w = waters(216, 21, 4.0)
    state = start([w])
    out = []
    for period in (0, -1):
        nb = Nonbonded(w[0], skin=0.05, list_period=period)
        out.append(run(nb, state, 40))
        nb.close()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1]) and out[0][2:] == out[1][2:]


def test_grouped_handle_does_not_keep_an_earlier_period():
    """A handle that was ungrouped with a list period, made grouped without one, follows the schedule
    of a handle made grouped in the first place (no rebuild while no site has moved half the skin)."""
    ws = [waters(300, 31, 4.0), waters(216, 32, 4.0)]
    state, systems = start(ws), [s for s, _ in ws]
    fresh = Nonbonded(systems, skin=1.0, list_period=0, groups=2)
    want = run(fresh, state, 40)
    used = Nonbonded(systems, skin=1.0, list_period=7, groups=1)
    run(used, state, 8)
    for p in used._params:
        p.list_period = 0
    assert used.L.moil_nb_set_groups(used.h, 2) == 0
    assert used.L.moil_nb_init_batch(used.h, len(systems), used._reps) == 0
    assert used.groups() == fresh.groups() == 2
    got = run(used, state, 40)
    fresh.close()
    used.close()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and got[2:] == want[2:]


def test_grouped_steps_follow_the_ungrouped_schedule():
    """With a list period, replica groups and the whole batch rebuild at the same steps and give the same bits."""
    ws = [waters(216, 33, 4.0), waters(300, 34, 4.0), waters(260, 35, 4.0)]
    state, systems = start(ws), [s for s, _ in ws]
    out = []
    for groups in (1, 3):
        nb = Nonbonded(systems, skin=1.0, list_period=9, groups=groups)
        assert (nb.groups() > 1) == (groups > 1)
        out.append(run(nb, state, 40))
        nb.close()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1]) and out[0][2] == out[1][2]


def loop_against_single_steps(make, state, steps, dt):
    a = make()
    got = run(a, state, steps, dt)
    a.close()
    b = make()
    want = run(b, state, 1, dt, calls=steps)
    b.close()
    assert torch.isfinite(got[0]).all()
    assert (got[0] - want[0]).abs().max() <= 1e-6 and (got[1] - want[1]).abs().max() <= 1e-3
    assert all(abs(x - y) <= 1e-5 * abs(y) for x, y in zip(got[2], want[2])) and abs(got[3] - want[3]) <= 1e-5 * want[3]


@pytest.mark.parametrize("precision", [MOIL_NB_MIXED, MOIL_NB_FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("name", ["waters", "solute"])
def test_step_graphs_match_single_steps(name, precision):
    """The gradient as the step graph's integrator forms it, in both precisions, with atoms outside waters (which
    have correction terms and no rigid molecule) and without."""
    if name == "waters":
        state, s, dt = start([waters(216, 41, 4.0)]), waters(216, 41, 4.0)[0], 0.0005
    else:
        s, dt = S.config1(seed=7, n_solute=61, n_ions=7, n_waters=299, box=24.0), 0.00002    # (no bonded terms)
        rng = np.random.Generator(np.random.PCG64(4))
        v = rng.normal(0.0, 4.0, (s.npt, 3))
        w = s.npt - 3 * s.nwaters
        v[w:] = np.repeat(v[w::3], 3, axis=0)
        state = (torch.tensor(s.coor, device="cuda"), torch.tensor(v, device="cuda"),
                 torch.tensor(S.molecules(s)[1], device="cuda"))
        torch.cuda.synchronize()
    loop_against_single_steps(lambda: Nonbonded(s, precision=precision, skin=1.0, list_period=10), state, 25, dt)


def test_one_group_outruns_its_lists():
    """Fast waters in the first group only: the run goes back to its start in every group and is redone."""
    ws = [waters(300, 51, 4.0), waters(216, 52, 0.05)]
    systems = [s for s, _ in ws]

    def make():
        nb = Nonbonded(systems, skin=0.05, list_period=1000, groups=2)
        assert nb.groups() == 2
        return nb
    loop_against_single_steps(make, start(ws), 40, 0.0005)

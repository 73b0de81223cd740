"""Which steps of a trajectory rebuild the lists, and who decides it: no list period at all, replica
groups, and lists outrun in one group only.  The same schedule gives the same bits; other schedules
are held against one call per step."""
import numpy as np
import pytest

from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import Nonbonded

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

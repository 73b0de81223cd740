"""Step loops whose list rebuilds the host foresees (moil_nb_md_step with a list period): runs of 64
steps and their remainder, and lists that are outrun before their period ends, where the run is
redone with the device's decision.  Against one call per step: the same kernels on the same list
schedule, so the trajectories agree to the FP32 forces' rounding at least."""
import numpy as np
import pytest

from moil_fnrfd_gb300 import systems as S
from moil_fnrfd_gb300.nb import Nonbonded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,period,skin", [(1, 10, 1.0), (63, 7, 1.0), (64, 10, 1.0), (131, 10, 1.0), (40, 1000, 0.05)])
def test_step_runs_match_single_steps(steps, period, skin):
    torch = pytest.importorskip("torch")
    s = S.water_box(216, 18.62, 21)
    rng = np.random.Generator(np.random.PCG64(3))
    n = s.npt // 3
    v0 = torch.tensor(np.repeat(rng.normal(0.0, 4.0, (n, 3)), 3, axis=0), device="cuda")     # Å/ps, rigid translation
    m = torch.tensor(np.tile([15.9994, 1.008, 1.008], n), device="cuda")
    x0 = torch.tensor(s.coor, device="cuda")
    out = []
    for single in (False, True):
        nb = Nonbonded(s, skin=skin, list_period=period)
        x, v = x0.clone(), v0.clone()
        torch.cuda.synchronize()
        for _ in range(steps if single else 1):
            e, ek = nb.md_step(x.data_ptr(), v.data_ptr(), m.data_ptr(), 0.0005, 1 if single else steps)
        out.append((x, v, e[0]["e_total"], ek))
        nb.close()
    (xa, va, ea, ka), (xb, vb, eb, kb) = out
    assert torch.isfinite(xa).all() and (xa - xb).abs().max() <= 1e-6 and (va - vb).abs().max() <= 1e-3
    assert abs(ea - eb) <= 1e-5 * abs(eb) and abs(ka - kb) <= 1e-5 * kb

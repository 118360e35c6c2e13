"""The volume kernels at every order, with and without viscosity
models, against the oracle.  Their matrix-instruction contractions run the oracle's FMA chains
in the oracle's order, so the tolerance is zero.  The orders cover every remainder of their tiles:
lines per direction modulo 8 (4, 9, 16, 25, 36, 49, 64, 81), Gauss points modulo 4, and one or two
interior Lobatto points per lane."""
import numpy as np
import pytest

from dsem_b200 import mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["none", "ev", "les", "ev+les"])
@pytest.mark.parametrize("p", range(1, 9))
def test_every_order_and_model_matches_oracle(oracle_mod, p, model):
    from dsem_b200.solver import Solver
    box = mesh.Box(3, 2, 4, p)  # three different element widths
    q = mesh.perturbed_taylor_green(box, seed=p, amp=0.2)
    dt = 0.2 * mesh.dtcalc(box, q)
    phys = dict(re=200.0, **(dict(cmu=0.5, mumax=2.0, shock=1) if "ev" in model else {}))
    s = Solver(box.desc(), **phys)
    c = oracle_mod.Case.from_desc(box.desc())
    c.set_phys(**phys)
    s.upload(q)
    c.set_q(q)
    if "les" in model:
        s.set_les(0.1, 1e3)
        c.set_les(0.1, 1e3)
    s.step(dt, 2)
    c.step(0.0, dt, 2)
    assert np.array_equal(s.download(), c.get_q())
    assert np.array_equal(s.rhs(), c.rhs())
    s.close()


@pytest.mark.parametrize("model", ["none", "ev"])
@pytest.mark.parametrize("p", range(1, 9))
def test_every_order_on_curved_elements_matches_oracle(oracle_mod, p, model):
    """Full metrics: the general volume kernel, whose three fluxes and 15 gradient components
    follow the oracle's order too."""
    from dsem_b200.solver import Solver
    box = mesh.Box(2, 3, 2, p, warp=0.02)
    q = mesh.perturbed_taylor_green(box, seed=p, amp=0.2)
    dt = 0.2 * mesh.dtcalc(box, q)
    phys = dict(re=200.0, **(dict(cmu=0.5, mumax=2.0, shock=1) if model == "ev" else {}))
    s = Solver(box.desc(), **phys)
    c = oracle_mod.Case.from_desc(box.desc())
    c.set_phys(**phys)
    s.upload(q)
    c.set_q(q)
    s.step(dt, 2)
    c.step(0.0, dt, 2)
    assert np.array_equal(s.download(), c.get_q())
    assert np.array_equal(s.rhs(), c.rhs())
    s.close()

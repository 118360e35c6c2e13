"""The volume kernels against the oracle on meshes large enough for each launch shape of
csrc/dsem_shapes.h: one right-hand side and one step, bit for bit (the kernels run the oracle's FMA
chains in the oracle's order)."""
import numpy as np
import pytest

from dsem_b200 import mesh

pytestmark = pytest.mark.gpu


def _check(oracle_mod, box, model):
    from dsem_b200.solver import Solver
    q = mesh.perturbed_taylor_green(box, seed=int(box.orders[0]), amp=0.2)
    dt = 0.2 * mesh.dtcalc(box, q)
    phys = dict(re=200.0, **(dict(cmu=0.5, mumax=2.0, shock=1) if "ev" in model else {}))
    desc = box.desc()
    s = Solver(desc, **phys)
    c = oracle_mod.Case.from_desc(desc)
    c.set_phys(**phys)
    s.upload(q)
    c.set_q(q)
    if "les" in model:
        s.set_les(0.1, 1e3)
        c.set_les(0.1, 1e3)
    s.step(dt, 1)
    c.step(0.0, dt, 1)
    assert np.array_equal(s.download(), c.get_q())
    assert np.array_equal(s.rhs(), c.rhs())
    s.close()


@pytest.mark.parametrize("model", ["none", "ev", "les", "ev+les"])
def test_p4_between_two_and_four_elements_per_sm(oracle_mod, model):
    _check(oracle_mod, mesh.Box(10, 6, 5, 4), model)  # 300 elements


@pytest.mark.parametrize("model", ["none", "ev"])
@pytest.mark.parametrize("p,n", [(4, (7, 7, 3)), (4, (6, 5, 5)), (4, (8, 8, 7)), (5, (7, 6, 7)), (5, (10, 6, 5)),
                                 (5, (8, 8, 7))])
def test_full_metrics_at_p4_and_p5(oracle_mod, p, n, model):
    """Each side of the limits at 148 (p = 4), 296 (p = 5) and 444 elements."""
    _check(oracle_mod, mesh.Box(*n, p, warp=0.02), model)

"""The volume kernels against the oracle on meshes large enough for each launch shape of
csrc/dsem_shapes.h: one right-hand side and one step, bit for bit (the kernels run the oracle's FMA
chains in the oracle's order), and the kinetic energy and dissipation after it, from the gradients
that the step's last stage saved (SUM_TOL: sums of positive terms over at most 729 points and
600 elements, in two orders at worst: 2 * 1329 roundings of 2^-53)."""
import numpy as np
import pytest

from dsem_b200 import mesh

pytestmark = pytest.mark.gpu
SUM_TOL = 2 * 1329 * 2.0 ** -53


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
    s.diag(dt, first=True)  # the step saves its gradients
    s.step(dt, 1)
    c.step(0.0, dt, 1)
    assert np.array_equal(s.download(), c.get_q())
    got, ref = s.diag(dt, first=True), c.diag(dt, True)
    assert abs(got[0] - ref[0]) <= SUM_TOL * ref[0] and abs(got[2] - ref[2]) <= SUM_TOL * ref[2]
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


@pytest.mark.parametrize("model", ["none", "ev", "les"])
@pytest.mark.parametrize("p,n", [(3, (10, 10, 6)), (4, (10, 10, 6)), (5, (10, 6, 5)), (6, (6, 5, 5)), (7, (6, 5, 5)),
                                 (8, (6, 5, 5))])
def test_default_shape_of_full_launches(oracle_mod, p, n, model):
    """Axis-aligned elements just above the wide shape's limit (592, 592, 296, 148 elements)."""
    _check(oracle_mod, mesh.Box(*n, p), model)


@pytest.mark.parametrize("model", ["none", "ev"])
@pytest.mark.parametrize("p,n", [(3, (8, 8, 7)), (6, (6, 5, 5))])
def test_full_metrics_default_shape_of_full_launches(oracle_mod, p, n, model):
    """Curved elements above the wide shape's limit (444, 148 elements)."""
    _check(oracle_mod, mesh.Box(*n, p, warp=0.02), model)

"""Device memory of dsem_adjoint: what calls leave with their contexts, and how it comes back."""
import numpy as np
import pytest

from dsem_b200 import mesh

pytestmark = pytest.mark.gpu
KEEP = 16 << 30  # all contexts together (include/dsem_gpu.h)
SLACK = 64 << 20  # code and small allocations of the driver


def _case(n, p):
    box = mesh.Box(n, n, n, p)
    q = mesh.perturbed_taylor_green(box, seed=2, amp=0.2)
    return box, q, 0.2 * mesh.dtcalc(box, q)


def _solver(box, q):
    from dsem_b200.solver import Solver
    s = Solver(box.desc(), re=400.0)
    s.upload(q)
    return s


def _same(a, b):
    return a[0] == b[0] and a[2] == b[2] and np.array_equal(a[1], b[1])


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("n,p,steps,snapshots", [(3, 4, 4, 0), (5, 8, 20, 5), (8, 6, 30, 0)])
def test_memory_kept_between_gradients_is_bounded(n, p, steps, snapshots):
    """Eight contexts (2.25 GB each in the last case), two gradients each: equal results, at most
    KEEP held, and all of it back when they close."""
    box, q, dt = _case(n, p)
    s = _solver(box, q)
    ref = s.adjoint(dt, steps, 3, snapshots)  # loads the kernels
    s.close()
    start = _free()
    ctx = [_solver(box, q) for _ in range(8)]
    before = _free()
    for s in ctx * 2:  # the second time in buffers that hold what the first left in them
        assert _same(s.adjoint(dt, steps, 3, snapshots), ref)
        assert before - _free() <= KEEP + SLACK
    big = s.adjoint(dt, 2 * steps, 3, 0)  # a larger block for one of them
    assert _same(s.adjoint(dt, 2 * steps, 3, 0), big) and before - _free() <= KEEP + SLACK
    for s in ctx:
        s.close()
    assert start - _free() <= SLACK


def test_kept_memory_comes_back_for_other_allocations():
    """On a card with 1 GiB free, a second context's gradient (2.25 GB) and new contexts (0.7 GB each)
    get the memory that the first context keeps."""
    import torch
    box, q, dt = _case(8, 6)
    a, b = _solver(box, q), _solver(box, q)
    ref = a.adjoint(dt, 30, 3, 0)
    big = mesh.Box(16, 16, 16, 6).desc()
    ballast = torch.empty(_free() - (1 << 30), dtype=torch.uint8, device="cuda")
    try:
        assert _same(b.adjoint(dt, 30, 3, 0), ref)
        from dsem_b200.solver import Solver
        more = [Solver(big) for _ in range(3)]
        for s in more:
            s.close()
        assert _same(a.adjoint(dt, 30, 3, 0), ref)
    finally:
        del ballast
        torch.cuda.empty_cache()
    a.close()
    b.close()

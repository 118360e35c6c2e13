"""Device memory of dsem_adjoint: what a call leaves with its context, and that the results do not
depend on how its buffers were had."""
import numpy as np
import pytest

from dsem_b200 import mesh

pytestmark = pytest.mark.gpu
KEEP = 256 << 20  # what a context may keep between calls (include/dsem_gpu.h)


@pytest.mark.parametrize("n,p,steps,snapshots", [(3, 4, 4, 0), (5, 6, 12, 0), (8, 6, 30, 0), (5, 8, 20, 5)])
def test_memory_kept_between_gradients_is_bounded(n, p, steps, snapshots):
    import torch
    from dsem_b200.solver import Solver
    box = mesh.Box(n, n, n, p)
    q = mesh.perturbed_taylor_green(box, seed=2, amp=0.2)
    dt = 0.2 * mesh.dtcalc(box, q)

    def gradient(s):
        s.upload(q)
        return s.adjoint(dt, steps, 3, snapshots)

    first = Solver(box.desc(), re=400.0)
    gradient(first)  # loads the kernels
    first.close()
    s = Solver(box.desc(), re=400.0)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    J, g, lr, _ = gradient(s)
    assert free - torch.cuda.mem_get_info()[0] <= KEEP + (32 << 20)
    for _ in range(2):  # buffers that hold what the call before left in them
        J2, g2, lr2, _ = gradient(s)
        assert J2 == J and lr2 == lr and np.array_equal(g2, g)
    s.close()

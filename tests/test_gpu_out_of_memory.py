"""A plan that finds no room is refused, and the next call that fits runs: the failed
allocation's error must not turn up at a later launch check."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_call_after_a_refused_plan_runs():
    import torch
    from hqc_gb300 import make_solver
    from hqc_gb300._lib import HqcgbError
    from hqc_gb300.workloads import box
    xp = np.random.default_rng(2).uniform(0, box(2), (2, 3))
    small = make_solver(2, box(2), 1.4, "gth-szv", dft=True, n_grid=15)
    want = small(xp)[1].clone()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(HqcgbError, match="out of memory"):  # 8 GB
            make_solver(54, box(54), 1.4, "gth-dzvp", dft=True, xc="pbe", n_grid=81, forces=True)
        assert bool((small(xp)[1] == want).all())
    finally:
        del fill
        torch.cuda.empty_cache()
    assert bool((make_solver(2, box(2), 1.4, "gth-szv", dft=True, n_grid=15)(xp)[1] == want).all())

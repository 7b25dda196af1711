"""A device allocation that fails while a context that is set up already
changes to another size (the failure is made on the host)."""
import numpy as np
import pytest

from vehicleroutingproblem_b200 import _native as N
from vehicleroutingproblem_b200 import instances as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(60, 1800), (1800, 60), (700, 600)])
def test_failed_change_of_size_leaves_a_usable_context(sizes):
    import torch
    first, second = (I.uniform_instance(n, 3, 940 + n) for n in sizes)
    kw = dict(ants=32, cand_k=16, seed=4)
    with N.Context(0) as c, N.Context(0) as fresh:
        c.setup_instance(first, **kw)
        c.run(3)
        free0 = torch.cuda.mem_get_info()[0]
        c.debug_inject(1, 1)
        with pytest.raises(N.AcoError) as err:
            c.setup_instance(second, **kw)
        assert err.value.status == N.ACO_ERR_ALLOCATION
        assert torch.cuda.mem_get_info()[0] >= free0  # it takes nothing
        for use in (lambda: c.run(1), c.best, c.state, c.tau, lambda: c.enqueue_epochs(1)):
            with pytest.raises((N.AcoError, ValueError)):
                use()
        for inst in (second, first, second):
            c.setup_instance(inst, **kw)
            st = c.run(5)
            fresh.setup_instance(inst, **kw)
            want = fresh.run(5)
            assert st.global_best == want.global_best and np.array_equal(c.tau(), fresh.tau())

"""A wait limit of 0 polls ends an RBF solve with the timeout status, as it does every
other call that sums on the evaluation grid; the context works normally afterwards."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["cg_rbf", "minres_rbf"])
@pytest.mark.parametrize("n", [1, 1000])
def test_no_polls_allowed(cuda, solver, n):
    from vortexparticlemc_cuda_gb300 import phash as P
    from vortexparticlemc_cuda_gb300._lib import WAIT_LIMIT_DEFAULT, VpmcError
    rng = np.random.default_rng(n)
    pos = torch.from_numpy(rng.random((n, 2)).astype(np.float32)).cuda()
    b = torch.from_numpy(rng.normal(size=n).astype(np.float32)).cuda()
    solve = getattr(P, solver)
    ctx = P.context()
    want, _ = solve(pos, b, 0.1, max_iter=5, allow_unconverged=True)
    ctx.set_wait_limit(0)
    try:
        for _ in range(2):
            with pytest.raises(VpmcError) as e:
                solve(pos, b, 0.1, max_iter=5, allow_unconverged=True)
            assert e.value.status == 5   # VPMC_ERR_TIMEOUT
    finally:
        ctx.set_wait_limit(WAIT_LIMIT_DEFAULT)
    assert torch.equal(solve(pos, b, 0.1, max_iter=5, allow_unconverged=True)[0], want)

"""The scalar PPPM's grid kernels (csrc/potential.cu) where their paths change:
the gradient buffer by pairs of cells (even edges) and by cells, windows beyond
both ends, and the deposit with every mass on a lattice whose planes fall on
cell faces, where the hash cell and the nearest grid point may differ."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K", [(7, 1), (8, 4), (10, 0), (12, 1), (12, 2), (24, 1), (24, 3)])
def test_grids_of_lattice_masses(oracle, n, K):
    """Tolerances of the grids' parity tests: FP64 sums in another order
    (1e-13), and 1e-6 where the FP32 multigrid enters."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pppm_vortex_bouyant_flow_sample_b200.potential import PotentialFieldSolver
    rng = np.random.default_rng(n)
    N = 3000
    pos = np.zeros((N, 4), np.float32)
    pos[:, :3] = rng.integers(-8, 9, (N, 3)) / 16.0
    pos[0, :3], pos[1, :3] = -0.5, 0.5
    mass = rng.uniform(0.5, 1.5, N)
    dev = [torch.from_numpy(a).cuda() for a in (pos, mass)]
    s = PotentialFieldSolver()
    s.initializeSolver(n, n, n, K, N, N)
    s.setMassParameter(N, *dev)
    s.setEvalParameter(N, dev[0])
    s.computeFarFieldBuffer()
    got = {k: s.grids()[k].numpy() for k in ("density", "rhs", "far")}
    s.shutdown()
    d = oracle.potential(n, K, pos, mass, pos, dump=True)[1]
    assert rel_l2(got["density"], d["density"]) <= 1e-13
    assert rel_l2(got["rhs"], d["rhs"]) <= 1e-13
    assert rel_l2(got["far"], d["far"]) <= 1e-6

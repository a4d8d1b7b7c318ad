"""The grid kernels at the edges where they change.  The multigrid: the launch
that holds the levels of edge <= 32 (csrc/mg_tail.cu: slabs of 4 planes of a
level of edge 17 to 32, the level of edge 9 to 16 and the coarsest one), and
the fused red-black sweep of the larger levels (csrc/mg_sweep.cu: whole rows,
tiles of at most 16 of them, fewer above edge 256, chunks of planes), against
the oracle's FP64 schedule.

A solve ends with an FP64 defect correction whose FP32 cycle rounds relative
to the correction it computes: below 1e-6 of the solution (the bound of the
scene's potential in test_gpu_parity).  One V-cycle from a random x is all
correction: up to seven levels of 16 half sweeps and two transfers, each
rounding to 2^-24 of values of the correction's size with signs of their own,
sqrt(126) x 2^-24 = 7e-7 of it.  6e-6 is nine times that.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pb():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pppm_vortex_bouyant_flow_sample_b200 as pb
    pb.load()
    return pb


@pytest.mark.parametrize("n", [10, 12, 14, 16, 20, 24, 28, 32, 40, 48, 56, 64, 80, 112, 160, 320, 448])
def test_full_multigrid_and_vcycle(pb, oracle, n):
    import torch
    rng = np.random.default_rng(n)
    b = rng.standard_normal(n ** 3)
    mg = pb.MultiGridSolver3DPeriod_double()
    mg.m_InitialSystem(n, n, n)
    x = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
    mg.m_FullMultiGrid(x, torch.from_numpy(b).cuda())
    ref = oracle.mg_fmg(np.zeros(n ** 3), b, n)
    assert rel_l2(x.cpu().numpy(), ref) <= 1e-6
    x0 = rng.standard_normal(n ** 3)
    x = torch.from_numpy(x0.copy()).cuda()
    mg.m_Vcycle(x, torch.from_numpy(b).cuda())
    ref = oracle.mg_vcycle(x0, b, n)
    assert np.linalg.norm(x.cpu().numpy() - ref) <= 6e-6 * np.linalg.norm(ref - x0)
    mg.m_FinalMemoryEachLevel()


@pytest.mark.parametrize("n", [16, 32, 40, 64])
def test_vcycle_of_a_slice_at_an_odd_offset(pb, oracle, n):
    """x and b need only be aligned as doubles: edges whose last sweep adds to
    x by pairs of doubles (above 32) and edges that end in the cluster launch."""
    import torch
    rng = np.random.default_rng(n)
    x0, b = rng.standard_normal(n ** 3), rng.standard_normal(n ** 3)
    buf = torch.full((n ** 3 + 2,), 7.0, dtype=torch.float64, device="cuda")
    x = buf[1:-1]
    x.copy_(torch.from_numpy(x0))
    bb = torch.zeros(n ** 3 + 1, dtype=torch.float64, device="cuda")[1:]
    bb.copy_(torch.from_numpy(b))
    assert x.data_ptr() % 16 == 8 and bb.data_ptr() % 16 == 8
    mg = pb.MultiGridSolver3DPeriod_double()
    mg.m_InitialSystem(n, n, n)
    mg.m_Vcycle(x, bb)
    ref = oracle.mg_vcycle(x0, b, n)
    assert np.linalg.norm(x.cpu().numpy() - ref) <= 6e-6 * np.linalg.norm(ref - x0)
    assert buf[0].item() == 7.0 and buf[-1].item() == 7.0
    mg.m_FinalMemoryEachLevel()


@pytest.mark.parametrize("tol", [1e-6, 1e-10])
@pytest.mark.parametrize("n", [12, 16, 20, 28, 32, 40, 64, 112])
def test_corrected_cycles_reach_the_tolerance(pb, oracle, n, tol):
    """The solve to a tolerance: the residual of what it returns, in numpy's
    64 bits, and the number of cycles.  A cycle gains at least a factor 10
    (0.032 is the worst measured), so 10 of them reach 1e-10 from the first's."""
    import torch
    rng = np.random.default_rng(n)
    b = rng.standard_normal(n ** 3)
    mg = pb.MultiGridSolver3DPeriod_double()
    mg.m_InitialSystem(n, n, n)
    x = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
    rel = mg.m_FullMultiGrid(x, torch.from_numpy(b).cuda(), tol, pb.MG_CONVERGED, 10)
    mg.m_FinalMemoryEachLevel()
    r = b - oracle.apply_laplacian(x.cpu().numpy(), n)
    got = np.linalg.norm(r) / np.linalg.norm(b)
    assert got <= tol
    assert abs(rel - got) <= 1e-6 * got + 1e-14


@pytest.mark.parametrize("kind", ["constant", "dipole", "sine"])
@pytest.mark.parametrize("n", [16, 24, 64, 80])
def test_corrected_cycles_on_smooth_sources(pb, oracle, n, kind):
    """Sources whose solution lives on the coarse levels, where white noise
    (above) leaves little: 8 cycles, the first counting for two, at no more than
    a tenth each (0.032 is the worst measured) reach 1e-8 from any of them."""
    import torch
    c = (np.arange(n) + 0.5) / n
    z, y, x = np.meshgrid(c, c, c, indexing="ij")
    if kind == "constant":
        b = np.ones(n ** 3)
    elif kind == "sine":
        b = (np.sin(np.pi * x) * np.sin(2 * np.pi * y) * np.sin(np.pi * z)).ravel()
    else:
        b = np.zeros((n, n, n))
        b[n // 2, n // 2, 1], b[n // 2, n // 2, n - 2] = 1.0, -1.0
        b = b.ravel()
    mg = pb.MultiGridSolver3DPeriod_double()
    mg.m_InitialSystem(n, n, n)
    u = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
    mg.m_FullMultiGrid(u, torch.from_numpy(b).cuda(), 1e-8, pb.MG_CONVERGED, 8)
    mg.m_FinalMemoryEachLevel()
    r = b - oracle.apply_laplacian(u.cpu().numpy(), n)
    assert np.linalg.norm(r) <= 1e-8 * np.linalg.norm(b)


@pytest.mark.parametrize("n,K", [(n, K) for n in (10, 12, 20) for K in (-1, 0, 1, 2, 4)] +
                         [(40, 0), (48, 0), (160, 1), (160, 2)])
def test_far_field_grid(pb, oracle, n, K):
    """The far-field grid of the four-cell kernel (edges that are multiples of
    4, from 48 with K = 0: rows of 3 and 5 groups, windows beyond both ends, and
    of 40, which two blocks share) and of the one-cell kernel: FP32 sums of at
    most 728 terms beside an FP64 curl, so 1e-5."""
    import torch
    rng = np.random.default_rng(5)
    N = 900
    pos = np.zeros((N, 4), np.float32)
    pos[:, :3] = rng.uniform(0.0, 1.0, (N, 3))
    al = rng.normal(size=(N, 3))
    box = dict(fixed_origin=(0.0, 0.0, 0.0), fixed_length=1.0)
    scene = pb.Scene(n, K=K, cap_vort=N, cap_eval=N, domain="fixed", **box)
    scene.set_vortices(torch.from_numpy(pos).cuda(), torch.from_numpy(np.ascontiguousarray(al.T)).cuda())
    scene.build_far_field()
    far = scene.grid(pb.GRID_FAR).cpu().numpy()
    scene.close()
    d = oracle.pppm(oracle.params(n, K=K, domain_mode=1, **box), pos, al, pos[:4], None, 0, dump=True)[1]
    assert rel_l2(far, d["far_u"]) <= 1e-5

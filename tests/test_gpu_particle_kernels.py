"""The particle kernels at the sizes where their paths change: the sort in one
block and in tiles, the evaluation's warps and blocks
(one block's four warps share 32 points below a size), its dense and sparse
walks, and the deposit's cells."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

BOX = dict(fixed_origin=(0.0, 0.0, 0.0), fixed_length=1.0)


@pytest.fixture(scope="module")
def pb():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pppm_vortex_bouyant_flow_sample_b200 as pb
    pb.load()
    return pb


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _points(rng, N, lo=0.0, hi=1.0):
    p = np.zeros((N, 4), np.float32)
    p[:, :3] = rng.uniform(lo, hi, (N, 3))
    return p


@pytest.mark.parametrize("N", [1, 33, 2048, 2049, 4096, 4097, 8191, 8192, 8193, 12289])
@pytest.mark.parametrize("n", [8, 48])
def test_sort_is_stable_at_every_size(pb, n, N):
    """Keys ascending, equal keys in index order, every index once: the block
    sort (to 8,192 pairs, 2, 4 or 8 a thread), the tiles (4,096) and their
    remainders, two and three digits of key."""
    rng = np.random.default_rng(N)
    pm = pb.ParticleManager()
    pm.initSpatialHash(N, n, n, n)
    pm.setSpatialHashGrid(n, 1.0 / n, (0.0, 0.0, 0.0), N)
    pos = _points(rng, N)
    pm.doSpatialHash(_dev(pos), N)
    key, idx = pm.getHashTable().numpy(), pm.getIndexTable().numpy()
    pm.endSpatialHash()
    c = np.floor(pos[:, :3] / np.float32(1.0 / n)).astype(np.int64) % n
    want = (c[:, 2] * n + c[:, 1]) * n + c[:, 0]
    order = np.argsort(want, kind="stable")
    assert np.array_equal(idx, order)
    assert np.array_equal(key, want[order])


@pytest.mark.parametrize("K", [0, 1, 3, 4])
@pytest.mark.parametrize("a_cells", [0.0, 1.0])
@pytest.mark.parametrize("M", [1, 15, 16, 17, 32, 33, 129, 700])
def test_evaluation_of_few_points(pb, oracle, M, a_cells, K):
    """Ragged groups, warps and blocks of targets in a dense part of a scene (45
    vortices a cell), with the smoothing polynomial (a = 0.3 is 5 cells) and
    the exp form; the pair count leaves out lanes without a point."""
    rng = np.random.default_rng(M)
    N = 20000
    pos, al = _points(rng, N, 0.3, 0.7), rng.normal(size=(N, 3))
    ev = _points(rng, M, 0.25, 0.75)
    scene = pb.Scene(16, K=K, a=0.3, a_cells=a_cells, cap_vort=N, cap_eval=M, domain="fixed", **BOX)
    scene.set_vortices(_dev(pos), _dev(al.T))
    scene.build_far_field()
    u = scene.eval(_dev(ev)).cpu().numpy()
    pairs = scene.count_pairs(_dev(ev))
    a = scene.smoothing()
    scene.close()
    ref, d = oracle.pppm(oracle.params(16, K=K, a=a, domain_mode=1, **BOX), pos, al, ev, None, 0, dump=True)
    assert pairs == int(d["pairs"][0])
    assert rel_l2(u, ref) <= 1e-5


@pytest.mark.parametrize("M", [1, 32, 33, 127, 128, 129, 700])
def test_far_field_only_evaluation(pb, oracle, M):
    """K = -1 takes whole blocks of points at every size, alone and in a batch
    beside a scene with a near field (32 points a block)."""
    rng = np.random.default_rng(M)
    n, N = 16, 3000
    pos, al, ev = _points(rng, N), rng.normal(size=(N, 3)), _points(rng, M, -0.05, 1.05)
    jobs, want = [], []
    for K in (-1, 1):
        scene = pb.Scene(n, K=K, a=0.3, cap_vort=N, cap_eval=M, domain="fixed", **BOX)
        jobs.append((scene, _dev(pos), _dev(al.T), _dev(ev), None, 0))
        want.append(oracle.pppm(oracle.params(n, K=K, a=0.3, domain_mode=1, **BOX), pos, al, ev, None, 0)[0])
    batch = [u.cpu().numpy() for u in pb.batch_run(jobs)]
    scene = jobs[0][0]
    scene.set_vortices(*jobs[0][1:3])
    scene.build_far_field()
    alone = scene.eval(jobs[0][3]).cpu().numpy()
    for got, ref in ((alone, want[0]), (batch[0], want[0]), (batch[1], want[1])):
        assert rel_l2(got, ref) <= 1e-5
    for j in jobs:
        j[0].close()


@pytest.mark.parametrize("per_cell", [0.3, 2.0, 6.0, 20.0])
@pytest.mark.parametrize("seg", [0, 1])
def test_evaluation_from_sparse_to_dense(pb, oracle, per_cell, seg):
    """Groups of targets that span several cells walk their own boxes, dense
    ones the shared walk, with and without a segment's other end."""
    rng = np.random.default_rng(7)
    n = 24
    N = int(per_cell * (n - 4) ** 3)
    pos, al = _points(rng, N, 2.0 / n, 1.0 - 2.0 / n), rng.normal(size=(N, 3))
    other = pos.copy()
    ev = pos.copy()
    if seg:
        ev[:, :3] += rng.normal(0.0, 0.1 / n, (N, 3)).astype(np.float32)
    sub = np.sort(rng.choice(N, min(N, 3000), replace=False))
    scene = pb.Scene(n, a_cells=1.0, cap_vort=N, cap_eval=N, domain="fixed", **BOX)
    scene.set_vortices(_dev(pos), _dev(al.T))
    scene.build_far_field()
    u = scene.eval(_dev(ev), _dev(other), 1).cpu().numpy()
    scene.close()
    ref = oracle.pppm(oracle.params(n, a=float(np.float32(1.0 / n)), domain_mode=1, **BOX), pos, al, ev[sub],
                      other[sub], 1)[0]
    assert rel_l2(u[sub], ref) <= 1e-5


@pytest.mark.parametrize("a_cells", [0.0, 1.0])
@pytest.mark.parametrize("seg", [0, 1])
@pytest.mark.parametrize("M", [1000, 270000])
def test_points_without_a_near_field_leave_the_others_alone(pb, oracle, M, seg, a_cells):
    """Points at infinity, far outside the grid or not a number, which the
    evaluation order puts next to points at the grid's faces (a block's warps
    sharing a walk and not): those have their values, a point outside has
    none.  Far-field interpolation as everywhere, hence the same 1e-5."""
    rng = np.random.default_rng(M + seg)
    n, N = 16, 20000
    pos, al = _points(rng, N), rng.normal(size=(N, 3))
    ev = _points(rng, M, 0.001, 0.999)
    odd = np.arange(M) % 20
    bad = odd < 5
    ev[odd == 0, 0] = np.inf
    ev[odd == 1, 1] = -np.inf
    ev[odd == 2, :3] = 1e30
    ev[odd == 3, 2] = np.nan
    ev[odd == 4, 0] += 3.0
    other = ev.copy()
    other[:, 1] += np.float32(0.2 / n)
    scene = pb.Scene(n, K=1, a=0.3, a_cells=a_cells, cap_vort=N, cap_eval=M, domain="fixed", **BOX)
    scene.set_vortices(_dev(pos), _dev(al.T))
    scene.build_far_field()
    u = scene.eval(_dev(ev), _dev(other), seg).cpu().numpy()
    a = scene.smoothing()
    scene.close()
    sub = np.flatnonzero(~bad)[:1000]
    ref = oracle.pppm(oracle.params(n, K=1, a=a, domain_mode=1, **BOX), pos, al, ev[sub], other[sub], seg)[0]
    assert rel_l2(u[sub], ref) <= 1e-5
    assert np.isfinite(u[~bad]).all()
    assert (u[bad & (odd != 3)] == 0.0).all()


def test_deposit_of_uneven_cells(pb, oracle):
    """Rows of cells with none, one and hundreds of vortices, and vortices on
    cell faces (whose nearest cell may not be their hash cell)."""
    rng = np.random.default_rng(13)
    n = 20
    dense = (np.array([3, 10, 10]) + rng.uniform(0, 1, (3000, 3)) * np.array([12, 1, 1])) / n
    faces = rng.integers(1, n, (500, 3)) / n
    pos = np.zeros((3500, 4), np.float32)
    pos[:, :3] = np.concatenate([dense, faces])
    al = rng.normal(size=(3500, 3))
    scene = pb.Scene(n, cap_vort=3500, cap_eval=1, domain="fixed", **BOX)
    scene.set_vortices(_dev(pos), _dev(al.T))
    scene.build_far_field()
    got = scene.grid(pb.GRID_VORT).cpu().numpy()
    scene.close()
    d = oracle.pppm(oracle.params(n, domain_mode=1, **BOX), pos, al, pos[:4], None, 0, dump=True)[1]
    assert rel_l2(got, d["grid_vort"]) <= 1e-6

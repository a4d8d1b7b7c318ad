"""The particle kernels at the sizes where their paths change: the sort in one
block and in tiles, and the deposit of cells with very different numbers of
vortices."""
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

"""The particle kernels at the sizes where their paths change: the deposit of
cells with very different numbers of vortices."""
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

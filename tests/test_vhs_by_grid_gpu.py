"""Two grids as one launch per grid (tile BY_GRID of a VHSCollider): the same
launches, bitwise, as a collider of each grid alone; batches in any order and
several per grid; a device list on the first batch; and what the tuner stores."""
import numpy as np
import pytest
import torch

from helpers import mixed_maxwellians, vhs_cfg

pytestmark = pytest.mark.gpu


def _grids():
    from frfs_b200.backend import CUDABackend
    from frfs_b200.scattering import VHSGrid, vhs_prefactor
    from frfs_b200.velocitymesh import DGFSVelocityMesh
    grids, fs = [], []
    for Nv, mass in ((24, 1.0), (32, 2.0)):
        cfg = vhs_cfg(Nv, 4, 12, 6)
        be = CUDABackend(cfg)
        vm = DGFSVelocityMesh(be, cfg)
        gam, pref, _ = vhs_prefactor(vm, 0.81, 4.17e-10, 273.0, mass=mass)
        grids.append(VHSGrid(Nv, vm.L(), vm.qz(), vm.qw(), vm.sz(), vm.sw(), gam, pref, vm.cw(), vm.c0(),
                             torch.float32, be.device))
        rng = np.random.default_rng(Nv)
        fs.append(torch.from_numpy(np.stack([mixed_maxwellians(vm.cv(), rng) for _ in range(6)])).float().cuda())
    return grids, fs


def test_by_grid_equals_each_alone(cuda):
    from frfs_b200.autotune import tuned_alone
    from frfs_b200.scattering import BY_GRID, VHSCollider
    grids, fs = _grids()
    want = []
    for g, f in zip(grids, fs):
        q = torch.empty_like(f)
        VHSCollider([tuned_alone(g, f.device)], f.device)([(0, f, q, None)])
        want.append(q)
    for g in grids:
        g.struct.tile = BY_GRID
    both = VHSCollider(grids, cuda)
    q = [torch.full_like(f, float('nan')) for f in fs]
    both([(1, fs[1], q[1], None), (0, fs[0], q[0], None)])
    assert torch.equal(q[0], want[0]) and torch.equal(q[1], want[1])
    # one grid of the set alone, and two batches of one grid
    one = VHSCollider([grids[1]], cuda)
    q = torch.empty_like(fs[1])
    one([(0, fs[1], q, None)])
    assert torch.equal(q, want[1])
    a, b = torch.empty_like(fs[0]), torch.empty_like(fs[0][:2])
    both([(0, fs[0], a, None), (0, fs[0][:2].contiguous(), b, None)])
    assert torch.equal(a, want[0]) and torch.equal(b, want[0][:2])
    # the device list applies to the first batch only
    idx = torch.tensor([3, 1], dtype=torch.int32, device=cuda)
    cnt = torch.tensor([1], dtype=torch.int64, device=cuda)
    q = [torch.zeros_like(f) for f in fs]
    both([(1, fs[1], q[1], None), (0, fs[0], q[0], None)], index=idx, count=cnt)
    assert torch.equal(q[1][3], want[1][3])
    assert not bool(q[1][[0, 1, 2, 4, 5]].any()) and torch.equal(q[0], want[0])


def test_tuner_tries_one_launch_per_grid(cuda, monkeypatch, tmp_path):
    from frfs_b200 import autotune
    from frfs_b200.scattering import BY_GRID, VHSCollider
    monkeypatch.setattr(autotune, '_CACHE', str(tmp_path / 'tune.json'))
    grids, fs = _grids()
    rec = {}
    tile = autotune.tune_vhs(grids, cuda, reps=1, record=rec)
    assert 'by-grid' in rec['ms'] and all(g.struct.tile == tile for g in grids)
    best = min(rec['ms'], key=rec['ms'].get)
    assert (tile == BY_GRID) == (best == 'by-grid')
    again, _ = _grids()
    assert autotune.tune_vhs(again, cuda) == tile                     # from the cache
    q = [torch.empty_like(f) for f in fs]
    VHSCollider(again, cuda)([(0, fs[0], q[0], None), (1, fs[1], q[1], None)])
    assert all(bool(torch.isfinite(x).all()) for x in q)


@pytest.mark.parametrize('by_grid', [False, True])
def test_bad_lists_are_refused_before_any_launch(cuda, by_grid):
    """A grid index outside the set, an empty list, too many batches, and a bad
    second batch: the same errors in one launch and in one per grid, and nothing
    written."""
    from frfs_b200 import _lib
    from frfs_b200.scattering import BY_GRID, VHSCollider
    grids, fs = _grids()
    for g in grids:
        g.struct.tile = BY_GRID if by_grid else 0
    col = VHSCollider(grids, cuda)
    q = [torch.full_like(f, 7.0) for f in fs]
    good = (0, fs[0], q[0], None)
    bad = [([good, (2, fs[1], q[1], None)], IndexError), ([good, (-1, fs[1], q[1], None)], _lib.BdgfsError),
           ([], _lib.BdgfsError), ([good] * 5, _lib.BdgfsError),
           ([good, (1, fs[1], q[1].double(), None)], TypeError),
           ([good, (1, fs[1][:, ::2], q[1], None)], ValueError),
           ([good, (1, fs[1], q[1][:3], None)], ValueError)]
    for batches, err in bad:
        with pytest.raises(err):
            col(batches)
    torch.cuda.synchronize()
    assert all(bool((x == 7.0).all()) for x in q)


def test_c_entry_points_take_a_set_tuned_by_grid(cuda):
    """Grids that the tuner marked BY_GRID are still a valid argument of the C
    entry points: one launch, as with tile 0."""
    from frfs_b200 import _lib
    from frfs_b200.scattering import BY_GRID
    grids, fs = _grids()
    L, out = _lib.lib(), []
    for tile in (0, BY_GRID):
        for g in grids:
            g.struct.tile = tile
        arr = (_lib.VhsGrid * 2)(*[g.struct for g in grids])
        nb = L.bdgfs_vhs_scratch_bytes(arr, 2, 0)
        assert nb > 0
        scratch = torch.empty(nb, dtype=torch.uint8, device=cuda)
        counter = torch.zeros(1, dtype=torch.int64, device=cuda)
        for static in (False, True):
            q = [torch.full_like(f, float('nan')) for f in fs]
            bs = (_lib.VhsBatch * 2)(*[_lib.VhsBatch(grid=i, ndof=6, f=fs[i].data_ptr(), Q=q[i].data_ptr())
                                       for i in (0, 1)])
            if static:
                rc = L.bdgfs_vhs_collide_static(arr, 2, bs, 2, 1, _lib.stream_ptr())
            else:
                rc = L.bdgfs_vhs_collide(arr, 2, bs, 2, 1, _lib.ptr(scratch), nb, _lib.ptr(counter),
                                         _lib.stream_ptr())
            assert rc == 0
            torch.cuda.synchronize()
            out.append(q)
    for q in out[1:]:
        assert all(torch.equal(a, b) for a, b in zip(q, out[0]))
    arr[0].tile = -2
    assert L.bdgfs_vhs_scratch_bytes(arr, 2, 0) == 0

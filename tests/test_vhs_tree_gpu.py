"""The shift-tree form of the 24^3 and 32^3 FP32 collision kernels: direction sets
with every kind of tree node, work split over radii, ragged lists, and rows that
are not 16-byte aligned.

Reference: the FP64 oracle (<= 1e-3 of Q and 1e-5 of the loss term, the bounds
of the other FP32 variants).  A distribution has the same bits whole or cut over
radii, wherever it stands in a list, however many CTAs run, on and off a 16-byte
boundary and in place: runs that differ in these only are compared with
torch.equal."""
import numpy as np
import pytest
import torch

from helpers import mixed_maxwellians, oracle_for, rel_l2, vhs_cfg

pytestmark = pytest.mark.gpu

TREE = 10                               # tile index among the 24^3 FP32 variants
TILES = {24: TREE, 32: 3}


def _setup(Nrho, M, ssrule=None, Nv=24):
    from frfs_b200.backend import CUDABackend
    from frfs_b200.scattering import DGFSVHSGLLScatteringModel
    from frfs_b200.velocitymesh import DGFSVelocityMesh
    cfg = vhs_cfg(Nv, Nrho, M, 6, extra=f'tile = {TILES[Nv]}')
    if ssrule:
        cfg.set('spherical-design-rule', 'ssrule', str(ssrule))
    be = CUDABackend(cfg)
    vm = DGFSVelocityMesh(be, cfg)
    return be, vm, DGFSVHSGLLScatteringModel(be, cfg, vm)


def _rows(vm, n, seed=5):
    rng = np.random.default_rng(seed)
    return torch.from_numpy(np.stack([mixed_maxwellians(vm.cv(), rng) for _ in range(n)])).float().cuda()


grids = pytest.mark.parametrize('Nv', [24, 32])


def _check(vm, f, q, rows):
    orc = oracle_for(vm)
    for i in rows:
        F = f[i].double().cpu().numpy()
        Qo, got = orc.Q(F), q[i].double().cpu().numpy()
        assert rel_l2(got, Qo) < 1e-3, i
        assert np.linalg.norm(got - Qo) < 1e-5 * np.linalg.norm(orc.gain_loss(F)[1]), i


def _design(tmp_path, half):
    half = np.asarray(half, float)
    half = half / np.linalg.norm(half, axis=1, keepdims=True)
    p = tmp_path / 'design.txt'
    np.savetxt(p, np.concatenate([half, -half]), fmt='%.17g')
    return p


RNG = np.random.default_rng(0)
DESIGNS = {
    # no shared component: as many nodes and leaves as directions
    'generic': RNG.normal(size=(5, 3)),
    # one x-node; y-nodes with a mirrored leaf pair, an unmirrored one, and
    # two leaves; opposite and repeated directions; zero components
    'shared': [(1, .5, .7), (1, .5, -.7), (1, -.5, .7), (-1, -.5, .9 - .2), (1, .5, .7), (0, 0, 1),
               (0, 1, 0), (0, -1, 0), (1, 0, 0), (0, .6, .8), (0, .6, -.8)],
    'largest': RNG.normal(size=(48, 3)),
}


@grids
@pytest.mark.parametrize('name', list(DESIGNS))
def test_direction_trees(cuda, tmp_path, name, Nv):
    half = DESIGNS[name]
    be, vm, sm = _setup(4 if Nv == 24 else 2, len(half), _design(tmp_path, half), Nv)
    f = _rows(vm, 2)
    q = torch.full_like(f, float('nan'))
    sm.collide(f, q, project=False)
    _check(vm, f, q, (0, 1))


@grids
def test_too_many_directions_has_no_tree(cuda, tmp_path, Nv):
    from frfs_b200.autotune import variants
    half = np.random.default_rng(1).normal(size=(49, 3))
    cfg_path = _design(tmp_path, half)
    be, vm, sm48 = _setup(2, 12, Nv=Nv)
    from frfs_b200.scattering import VHSGrid
    sz = np.loadtxt(cfg_path)[:49]
    g = VHSGrid(Nv, vm.L(), vm.qz(), vm.qw(), sz, vm.sw(), 0.38, 1.0, vm.cw(), vm.c0(), torch.float32, be.device)
    assert len(variants([g])) == len(variants([sm48.grid])) - 1


@grids
@pytest.mark.parametrize('M', [12, 6])
@pytest.mark.parametrize('n', [1, 13, 75, 149, 297])
def test_split_over_radii_agrees(cuda, M, n, Nv):
    """Short lists and the last round of long ones cut the radii into parts (1
    row: one part per radius; others fewer, or none).  Of 600 rows, 592 are whole
    on 148 SMs and 8 are cut: every row has the bits of the short list."""
    be, vm, sm = _setup(12 if Nv == 24 else 5, M, Nv=Nv)
    f = _rows(vm, 8)[torch.arange(n) % 8].contiguous()
    q = torch.full_like(f, float('nan'))
    mom = torch.full((n, 10), float('nan'), dtype=torch.float64, device=f.device)
    sm.collide(f, q, moments=mom)
    rows = torch.arange(600) % n
    big = f[rows].contiguous()
    qb = torch.empty_like(big)
    sm.collide(big, qb)
    assert torch.equal(qb, q[rows])
    assert torch.isfinite(mom).all() and float(mom[:, 5:].abs().max()) < 1e-12
    # the same launch again
    q2 = torch.empty_like(q)
    sm.collide(f, q2)
    assert torch.equal(q, q2)
    if n == 1:
        sm.collide(f, q, project=False)
        _check(vm, f, q, (0,))


@grids
def test_device_list_and_unaligned_rows(cuda, Nv):
    """A device index list with a device count (the split follows the count),
    entries out of range skipped; rows at a 4-byte offset; in place."""
    be, vm, sm = _setup(12 if Nv == 24 else 5, 12, Nv=Nv)
    n3 = Nv**3
    f = _rows(vm, 8)[torch.arange(40) % 8].contiguous()
    want = torch.empty_like(f)
    sm.collide(f, want)
    idx = torch.tensor([31, 2, 17, -1, 40, 5], dtype=torch.int32, device=f.device)
    for count in (0, 1, 6):
        q = torch.zeros_like(f)
        cnt = torch.tensor([count], dtype=torch.int64, device=f.device)
        sm.collider([(0, f, q, None)], index=idx, count=cnt)
        done = [i for i in idx[:count].tolist() if 0 <= i < 40]
        for i in range(40):
            if i in done:
                assert torch.equal(q[i], want[i])
            else:
                assert not bool(q[i].any())
    g = torch.empty(3 * n3 + 1, device=f.device)[1:].view(3, n3)
    g.copy_(f[:3])
    q = torch.empty(3 * n3 + 1, device=f.device)[1:].view(3, n3)
    assert g.data_ptr() % 16 == 4
    sm.collide(g, q)
    assert torch.equal(q, want[:3])
    h = f[:3].clone()
    sm.collide(h, h)
    assert torch.equal(h, want[:3])


@grids
def test_scratch_limits(cuda, Nv):
    """One CTA's scratch is enough; less than a slot is refused."""
    import ctypes as C
    from frfs_b200 import _lib
    be, vm, sm = _setup(12 if Nv == 24 else 5, 12, Nv=Nv)
    f = _rows(vm, 5)
    want, q = torch.empty_like(f), torch.full_like(f, float('nan'))
    sm.collide(f, want)
    arr = (_lib.VhsGrid * 1)(sm.grid.struct)
    bs = (_lib.VhsBatch * 1)(_lib.VhsBatch(grid=0, ndof=5, f=f.data_ptr(), Q=q.data_ptr()))
    counter = torch.zeros(1, dtype=torch.int64, device=f.device)
    per = _lib.lib().bdgfs_vhs_scratch_bytes(arr, 1, 1)
    s = torch.empty(per, dtype=torch.uint8, device=f.device)
    call = lambda n: _lib.lib().bdgfs_vhs_collide(arr, 1, bs, 1, 1, s.data_ptr(), C.c_size_t(n),
                                                  counter.data_ptr(), _lib.stream_ptr())
    assert call(per) == 0
    assert torch.equal(q, want)
    assert call(1024) == -5


@pytest.mark.parametrize('Nv,old,new', [(24, 9, TREE), (32, 2, 3)])
def test_a_launch_with_nothing_to_do_is_short(cuda, Nv, old, new):
    """A device list whose count is zero (the fallback list of every hybrid call)
    costs no more than twice what the variants without a direction tree take for
    it: the kernel leaves before it builds the tree.  Device time of launches in
    a graph."""
    from frfs_b200.scattering import VHSCollider
    be, vm, sm = _setup(12, 12, Nv=Nv)
    f = torch.zeros(64, Nv**3, device=cuda)
    q = torch.full_like(f, 7.0)
    idx = torch.zeros(64, dtype=torch.int32, device=cuda)
    cnt = torch.zeros(1, dtype=torch.int64, device=cuda)

    def per_launch(tile):
        sm.grid.struct.tile = tile
        col = VHSCollider([sm.grid], be.device)
        run = lambda: col([(0, f, q, None)], index=idx, count=cnt)
        run()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(50):
                run()
        best = 1e30
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.replay()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 20.0)
        return best
    t_old, t_new = per_launch(old), per_launch(new)
    print(f'{Nv}^3: empty launch {t_old:.2f} us, with a tree {t_new:.2f} us')
    assert t_new < 2 * t_old
    assert bool((q == 7.0).all())

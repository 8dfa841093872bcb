"""The small-grid collision kernel (Nyquist term from its planes) against the
FP64 oracle: every grid size and precision, one to several batches of
directions, with and without the exact term, short lists cut over radii, device
lists.

A distribution has the same bits whole or cut over radii and wherever it stands in a
list (torch.equal).  FP64 with the exact term: 1e-10 of Q; without it, the variants agree with each
other to 1e-12; FP32: 1e-3 of Q and 1e-5 of the loss term (the bounds of the
other variants)."""
import numpy as np
import pytest
import torch

from helpers import mixed_maxwellians, oracle_for, rel_l2, vhs_cfg

pytestmark = pytest.mark.gpu


def _setup(Nv, Nrho, M, prec, ssrule=None):
    from frfs_b200.autotune import variants
    from frfs_b200.backend import CUDABackend
    from frfs_b200.scattering import DGFSVHSGLLScatteringModel, VHSCollider
    from frfs_b200.velocitymesh import DGFSVelocityMesh
    cfg = vhs_cfg(Nv, Nrho, M, 5, precision=prec, extra='tile = 0')
    if ssrule:
        cfg.set('spherical-design-rule', 'ssrule', str(ssrule))
    be = CUDABackend(cfg)
    vm = DGFSVelocityMesh(be, cfg)
    sm = DGFSVHSGLLScatteringModel(be, cfg, vm)
    old = sm.collider
    sm.grid.struct.tile = len(variants([sm.grid])) - 1
    sm.collider = VHSCollider([sm.grid], be.device)
    return be, vm, sm, old


def _rows(vm, n, be):
    rng = np.random.default_rng(17)
    return torch.from_numpy(np.stack([mixed_maxwellians(vm.cv(), rng) for _ in range(n)])).to(be.fpdtype).to(be.device)


@pytest.mark.parametrize('Nv', [8, 12, 16])
@pytest.mark.parametrize('prec', ['single', 'double'])
@pytest.mark.parametrize('M', [1, 3, 6, 7, 12])
def test_exact_kernel_parity(cuda, tmp_path, Nv, prec, M):
    rule = None
    if M == 7:                               # a second, short batch of directions
        half = np.random.default_rng(4).normal(size=(7, 3))
        half /= np.linalg.norm(half, axis=1, keepdims=True)
        rule = tmp_path / 'design.txt'
        np.savetxt(rule, np.concatenate([half, -half]), fmt='%.17g')
    be, vm, sm, old = _setup(Nv, 3, M, prec, rule)
    f = _rows(vm, 2, be)
    q, w = torch.full_like(f, float('nan')), torch.empty_like(f)
    sm.collide(f, q, project=False, exact=True)
    orc = oracle_for(vm)
    for i in range(2):
        F, got = f[i].double().cpu().numpy(), q[i].double().cpu().numpy()
        want = orc.Q(F)
        if prec == 'double':
            assert rel_l2(got, want) < 1e-10
        else:
            assert rel_l2(got, want) < 1e-3
            assert np.linalg.norm(got - want) < 1e-5 * np.linalg.norm(orc.gain_loss(F)[1])
    # without the term: the other variants' result
    sm.collide(f, q, project=False, exact=False)
    tile, sm.grid.struct.tile = sm.grid.struct.tile, 0
    old([(0, f, w, None)], project=False, exact=False)
    sm.grid.struct.tile = tile
    assert float((q - w).norm() / w.norm()) < (1e-12 if prec == 'double' else 5e-5)


@pytest.mark.parametrize('Nv,prec', [(8, 'single'), (12, 'double'), (16, 'single'), (16, 'double')])
@pytest.mark.parametrize('n', [1, 13, 75, 149, 500])
def test_exact_kernel_split(cuda, Nv, prec, n):
    be, vm, sm, _ = _setup(Nv, 8, 6, prec)
    base = _rows(vm, 6, be)
    f = base[torch.arange(n) % 6].contiguous()
    q = torch.full_like(f, float('nan'))
    mom = torch.full((n, 10), float('nan'), dtype=torch.float64, device=f.device)
    sm.collide(f, q, moments=mom, exact=True)
    big = base[torch.arange(3000) % 6].contiguous()
    w = torch.empty_like(big)
    sm.collide(big, w, exact=True)
    want = w[:6][torch.arange(n) % 6]
    assert torch.equal(q, want) and torch.equal(w, w[:6][torch.arange(3000) % 6])
    assert torch.isfinite(mom).all() and float(mom[:, 5:].abs().max()) < 1e-11
    q2 = torch.empty_like(q)
    sm.collide(f, q2, exact=True)
    assert torch.equal(q, q2)
    # a device list: the same rows, skipping entries out of range
    idx = torch.tensor([n - 1, 0, -3, n, n // 2], dtype=torch.int32, device=f.device)
    cnt = torch.tensor([4], dtype=torch.int64, device=f.device)
    r = torch.zeros_like(f)
    if n >= 5:
        sm.collider([(0, f, r, None)], index=idx, count=cnt, exact=True)
        done = [i for i in idx[:4].tolist() if 0 <= i < n]
        assert torch.equal(r[done], want[done])
        rest = [i for i in range(n) if i not in done]
        assert not bool(r[rest].any())


@pytest.mark.parametrize('prec', ['single', 'double'])
@pytest.mark.parametrize('Nv', [8, 12, 16])
def test_projection_of_every_variant(cuda, prec, Nv):
    """Every compiled variant conserves mass, momentum and energy, by sums taken
    outside the kernel, and gives the projected Q of the others.  The sums of Q
    over n values: FP64 n eps = 1e-12 of their sum of magnitudes; FP32 one
    rounding of each value (6e-8) at most.  Between variants: as without
    projection."""
    from frfs_b200.autotune import variants
    from frfs_b200.scattering import VHSCollider
    be, vm, sm, _ = _setup(Nv, 4, 6, prec)
    f = _rows(vm, 3, be)
    cv = vm.cv()
    phi = np.stack([np.ones(cv.shape[1]), *cv, np.sum(cv * cv, axis=0)])
    qs = []
    for t in range(len(variants([sm.grid]))):
        sm.grid.struct.tile = t
        q = torch.full_like(f, float('nan'))
        VHSCollider([sm.grid], be.device)([(0, f, q, None)], project=True, exact=True)
        Q = q.double().cpu().numpy()
        assert (np.abs(Q @ phi.T) <= (1e-12 if prec == 'double' else 1e-7) * (np.abs(Q) @ np.abs(phi).T)).all(), t
        qs.append(q.double())
        assert float((qs[-1] - qs[0]).norm() / qs[0].norm()) < (1e-12 if prec == 'double' else 5e-5), t

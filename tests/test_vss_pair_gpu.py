"""The two-species 24^3 FP32 mixture kernel (opposite directions share slices):
against the FP64 operator on the GPU (itself pinned to the oracle and to the
reference's kernels), for split and unsplit launches, few CTAs, direction sets
that the kernel does not apply to, and scratch limits.

FP32 against FP64: 2e-4 of Q, the bound of the other FP32 paths.  A distribution
has the same bits whole or cut over radii, wherever it stands in a list and
however many CTAs run: torch.equal.  The general kernel, which associates sums
differently: 1e-7 of the gain, amplified by Q's gain-loss cancellation (about 10 on
these states): 2e-5."""
import numpy as np
import pytest
import torch

from frfs_b200.backend import CUDABackend
from frfs_b200.dgfsbi import DGFSBiVelocityMesh, DGFSBiVSSGLLScatteringModel
from helpers import mixture, vss_cfg

pytestmark = pytest.mark.gpu


def _model(Nrho, M, precision='single', ssrule=None, Mpre=12, masses=(39.96e-3, 83.798e-3), project=False):
    cfg = vss_cfg(24, Nrho, M, Mpre, masses=masses, dev=6, precision=precision, project=project)
    if ssrule:
        cfg.set('spherical-design-rule', 'ssrule', str(ssrule))
    be = CUDABackend(cfg)
    vm = DGFSBiVelocityMesh(be, cfg, len(masses))
    return be, vm, DGFSBiVSSGLLScatteringModel(be, cfg, vm)


def _rows(vm, n, seed=3):
    rng = np.random.default_rng(seed)
    F = [mixture(vm.cv(), vm.masses(), rng) for _ in range(n)]
    return [torch.from_numpy(np.stack([f[p] for f in F])).float().cuda() for p in range(len(vm.masses()))]


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize('Nrho,M,masses', [(5, 12, (39.96e-3, 83.798e-3)), (4, 6, (39.96e-3, 20.18e-3)),
                                           (3, 2, (39.96e-3, 39.96e-3))])
def test_pair_matches_fp64(cuda, Nrho, M, masses):
    be, vm, sm = _model(Nrho, M, masses=masses)
    assert sm._pair is not None
    _, _, sm64 = _model(Nrho, M, precision='double', masses=masses)
    assert sm64._pair is None
    fs = _rows(vm, 3)
    Qs = [torch.full_like(f, float('nan')) for f in fs]
    sm.collide(fs, Qs)
    W = [torch.empty_like(f, dtype=torch.float64) for f in fs]
    sm64.collide([f.double() for f in fs], W)
    for q, w in zip(Qs, W):
        assert _rel(q, w) < 2e-4


@pytest.mark.parametrize('n,nctas', [(1, 148), (20, 148), (97, 148), (200, 148), (7, 2), (3, 1)])
def test_pair_split_and_few_ctas_agree(cuda, n, nctas):
    be, vm, sm = _model(6, 6)
    base = _rows(vm, 4)
    pick = torch.arange(n) % 4
    fs = [f[pick].contiguous() for f in base]
    sm._nctas, sm._scratch = nctas, None
    Qs = [torch.full_like(f, float('nan')) for f in fs]
    sm.collide(fs, Qs)
    big = torch.arange(600) % 4
    sm._nctas, sm._scratch = 148, None
    B = [f[big].contiguous() for f in base]
    W = [torch.empty_like(f) for f in B]
    sm.collide(B, W)
    for q, w in zip(Qs, W):
        assert torch.equal(q, w[:4][pick]) and torch.equal(w, w[:4][big])
    Q2 = [torch.empty_like(f) for f in fs]
    sm._nctas, sm._scratch = nctas, None
    sm.collide(fs, Q2)
    assert all(torch.equal(a, b) for a, b in zip(Qs, Q2))


def test_pair_needs_antipodal_halves(cuda, tmp_path):
    """The same directions in another order, three species, another grid: the
    general kernel, the same operator."""
    be, vm, sm = _model(4, 12)
    half = vm.sz()[:6]
    p = tmp_path / 'interleaved.txt'
    np.savetxt(p, np.stack([half, -half], 1).reshape(12, 3), fmt='%.17g')
    _, _, other = _model(4, 12, ssrule=p)
    assert other._pair is None
    fs = _rows(vm, 2)
    Q, W = [[torch.empty_like(f) for f in fs] for _ in range(2)]
    sm.collide(fs, Q)
    other.collide(fs, W)
    for q, w in zip(Q, W):
        assert _rel(q, w) < 2e-5
    _, _, three = _model(2, 2, masses=(39.96e-3, 83.798e-3, 20.18e-3))
    assert three._pair is None


@pytest.mark.parametrize('S', [1, 2, 3, 4])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('Nv,shift', [(16, 0), (24, 1), (7, 0)])
def test_projection_kernel(cuda, S, dtype, Nv, shift):
    """bdgfs_vss_project alone against the stacked least-squares projection
    (FP64 sums: n eps of the magnitudes; FP32 result: one rounding)."""
    import ctypes as C
    from frfs_b200 import _lib
    from frfs_b200.dgfsbi import mixture_gram_inverse
    from oracle.vss import project_mixture
    c0 = np.linspace(-5 + 5 / Nv, 5 - 5 / Nv, Nv)
    cv = np.stack([a.ravel() for a in np.meshgrid(c0, c0, c0, indexing='ij')])
    masses = [1.0, 2.1, 0.5, 1.3][:S]
    rng = np.random.default_rng(S)
    n, nd = Nv**3, 3
    Q = [torch.empty(nd * n + shift, dtype=dtype, device='cuda')[shift:].view(nd, n) for _ in range(S)]
    for q in Q:
        q.copy_(torch.from_numpy(rng.normal(size=(nd, n)) * np.exp(-np.sum(cv * cv, axis=0) / 4)))
    start = [q.double().cpu().numpy() for q in Q]
    f64 = lambda a: torch.as_tensor(np.asarray(a, np.float64)).cuda().contiguous()
    dc, dm, dg = f64(c0), f64(masses), f64(mixture_gram_inverse(c0, masses).ravel())
    a = _lib.VssProjArgs(Nv=Nv, nspcs=S, ndof=nd, fp64=int(dtype == torch.float64), c0=dc.data_ptr(),
                         mass=dm.data_ptr(), ginv=dg.data_ptr())
    for p in range(S):
        a.Q[p] = Q[p].data_ptr()
    assert _lib.lib().bdgfs_vss_project(C.byref(a), _lib.stream_ptr()) == 0
    for d in range(nd):
        want = project_mixture([s[d] for s in start], cv, masses)
        for p in range(S):
            got = Q[p][d].double().cpu().numpy()
            assert np.abs(got - want[p]).max() <= (1e-10 if dtype == torch.float64 else 2e-7) * np.abs(want[p]).max()


def test_pair_scratch_limits(cuda):
    import ctypes as C
    from frfs_b200 import _lib
    be, vm, sm = _model(2, 2)
    fs = _rows(vm, 2)
    Qs = [torch.empty_like(f) for f in fs]
    t = sm._pair
    a = _lib.VssPairArgs(Nv=24, Nrho=2, M=2, ndof=2, phase=t['phase'].data_ptr(), bself=t['bself'].data_ptr(),
                         bcross=t['bcross'].data_ptr(), c=t['c'].data_ptr())
    for p in (0, 1):
        a.f[p], a.Q[p] = fs[p].data_ptr(), Qs[p].data_ptr()
    L = _lib.lib()
    s = torch.empty(L.bdgfs_vss_pair_scratch_bytes(1), dtype=torch.uint8, device='cuda')
    call = lambda nb: L.bdgfs_vss_pair_collide(C.byref(a), s.data_ptr(), nb, _lib.stream_ptr())
    assert call(1000) == -5 and call(s.numel()) == 0
    a.M = 3
    assert call(s.numel()) == -1
    a.M, a.Nv = 2, 16
    assert call(s.numel()) == -3


def test_pair_scratch_follows_the_call(cuda):
    """A model holds what its largest call needs (a slot is 24 24^2 float4s: 221
    KB; a CTA has two, a radius of a cut distribution one), and a call in the
    least scratch gives the bits of a call in the most."""
    from frfs_b200 import _lib
    be, vm, sm = _model(6, 6)
    L, slot = _lib.lib(), 24**3 * 16
    most = L.bdgfs_vss_pair_scratch_bytes(sm._nctas)
    base = _rows(vm, 4)
    held = 0
    for n, slots in ((1, 6 * 2 + 6), (5, 30 * 2 + 30), (20, 120 * 2 + 120), (3, 0), (150, 148 * 2 + 12)):
        pick = torch.arange(n) % 4
        fs = [f[pick].contiguous() for f in base]
        Q, W = [[torch.full_like(f, float('nan')) for f in fs] for _ in range(2)]
        sm.collide(fs, Q)
        if sm._nctas == 148:
            held = max(held, slots * slot)                       # (grown by doubling)
            assert held <= sm._scratch.numel() <= 2 * held + 8192
        keep, sm._scratch = sm._scratch, torch.empty(most, dtype=torch.uint8, device='cuda')
        a = _lib.VssPairArgs(Nv=24, Nrho=6, M=6, ndof=n, phase=sm._pair['phase'].data_ptr(),
                             bself=sm._pair['bself'].data_ptr(), bcross=sm._pair['bcross'].data_ptr(),
                             c=sm._pair['c'].data_ptr())
        for p in (0, 1):
            a.f[p], a.Q[p] = fs[p].data_ptr(), W[p].data_ptr()
        _lib.check(L.bdgfs_vss_pair_collide(_lib.ref(a), sm._scratch.data_ptr(), most, _lib.stream_ptr()), 'pair')
        sm._scratch = keep
        assert all(torch.equal(q, w) for q, w in zip(Q, W))
    assert [L.bdgfs_vss_pair_scratch_for(*a) for a in ((0, 1, 1), (1, 0, 1), (1, 1, 0))] == [0, 0, 0]


@pytest.mark.parametrize('precision', ['single', 'double'])
def test_a_captured_call_keeps_its_scratch(cuda, precision):
    """A graph of a small call still works after a larger call has made the model's
    scratch grow: the memory that the graph writes to has not gone to others."""
    be, vm, sm = _model(4, 6, precision=precision)
    base = [f.to(be.fpdtype) for f in _rows(vm, 2)]
    want = [torch.empty_like(f) for f in base]
    sm.collide(base, want)
    first = sm._scratch.data_ptr(), sm._scratch.numel()
    got = [torch.empty_like(f) for f in base]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sm.collide(base, got)
    assert sm._scratch.data_ptr() == first[0]
    big = [f[torch.arange(40) % 2].contiguous() for f in base]
    sm.collide(big, [torch.empty_like(f) for f in big])
    assert sm._scratch.numel() > first[1]
    other = [torch.full((first[1],), 7, dtype=torch.uint8, device='cuda') for _ in range(4)]
    assert all(t.data_ptr() + t.numel() <= first[0] or first[0] + first[1] <= t.data_ptr() for t in other)
    g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert all(bool((t == 7).all()) for t in other)

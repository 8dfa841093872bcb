"""bdgfs_fr_rhs_affine against the dense residual (bdgfs_fr_rhs_gather /
bdgfs_fr_rhs, pinned to the oracle elsewhere): every shape it has, both
precisions, grids whose 4-velocity chunks hold both signs of a velocity
component (Nv = 10, 12, 6), sheared elements (every chunk may), every boundary
kind, rows without vector alignment, the in-place update, and combinations with
none, one or both of x1 and x2.

FP64 to 1e-12 and FP32 to 2e-5 of the result, the bounds of the other FR paths."""
import numpy as np
import pytest
import torch

from frfs_b200 import _lib
from frfs_b200.backend import CUDABackend
from frfs_b200.mesh import StructuredMesh
from frfs_b200.system import DGFSSystem
from helpers import bc_cfg, couette_cfg

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def coarse_grids(monkeypatch):
    """Wall Maxwellians on grids too coarse for the support check (FR does not
    care what the rows hold)."""
    from frfs_b200.initcond import DGFSMaxwellianInitCondition

    def rows(self):
        d2 = np.sum((self.vm.cv() - self._uini)**2, axis=0)
        self._init_vals = self._rhoini / (np.pi * self._Tini)**1.5 * np.exp(-d2 / self._Tini)
    monkeypatch.setattr(DGFSMaxwellianInitCondition, 'perform_precomputation', rows)


class Sheared(StructuredMesh):
    """The box's elements under a constant shear (still affine)."""

    def __init__(self, *a, **k):
        super().__init__(*a, **k)
        A = np.eye(self.ndims) + 0.3 * np.triu(np.ones((self.ndims, self.ndims)), 1)
        A[1, 0] = -0.2
        self.eles = self.eles @ A.T

    def pair_shift(self, e, f, e2, f2):
        A = np.eye(self.ndims) + 0.3 * np.triu(np.ones((self.ndims, self.ndims)), 1)
        A[1, 0] = -0.2
        return A @ super().pair_shift(e, f, e2, f2)


def _system(ndims, order, Nv, precision, sheared=False, bcs=None):
    if bcs:
        cfg = bc_cfg(Nv, order, bcs, precision=precision)
    else:
        cfg = couette_cfg(Nv, 4, 6, 5, order, precision=precision)
    cfg.set('scattering-model', 'tile', '0')
    if Nv not in (8, 12, 16, 24, 32):                  # no collision kernel: FR alone
        cfg.set('scattering-model', 'type', 'bgk-direct-gll')
        cfg.set('scattering-model', 'muRef', '2.117e-5')
    be = CUDABackend(cfg)
    cls = Sheared if sheared else StructuredMesh
    shape, hi = ((3, 4), (1.0, 0.5)) if ndims == 2 else ((2, 3, 2), (1.0, 0.5, 0.7))
    lo = (0.0, -0.5) if ndims == 2 else (0.0, -0.5, 0.0)
    per = '' if bcs else ('x' if ndims == 2 else 'xz')
    from frfs_b200.adgfs import ADGFSSystem
    s = (DGFSSystem if Nv in (8, 12, 16, 24, 32) else ADGFSSystem)(be, cls(shape, lo, hi, periodic=per), cfg, nreg=5)
    rng = np.random.default_rng(order * 100 + Nv)
    for u in s.eles_scal_upts_inb_full:
        u.copy_(torch.from_numpy(rng.normal(size=tuple(u.shape))).to(u))
    return s


def _both(s, uin, out, **kw):
    """advect_combine through the affine kernel and through the dense one."""
    res = []
    start = s._bank(out).clone()
    af, tp = s.ele.affine, s.ele.tensor
    assert af is not None
    for dense in (False, True):
        s._bank(out).copy_(start)
        if dense:
            s.ele.affine = s.ele.tensor = None
        s.advect_combine(0.0, uin, out, **kw)
        res.append(s._bank(out).double().clone())
    s.ele.affine, s.ele.tensor = af, tp
    s._bank(out).copy_(start)
    return res


def _tol(s):
    return 1e-12 if s.backend.fpdtype == torch.float64 else 2e-5


def _close(a, b, s):
    assert float((a - b).norm() / b.norm()) < _tol(s)


@pytest.mark.parametrize('ndims,order', [(2, 1), (2, 2), (2, 3), (3, 1), (3, 2)])
@pytest.mark.parametrize('Nv,precision', [(16, 'single'), (12, 'single'), (10, 'single'), (6, 'double'), (16, 'double')])
@pytest.mark.parametrize('sheared', [False, True])
def test_affine_equals_dense(cuda, ndims, order, Nv, precision, sheared):
    s = _system(ndims, order, Nv, precision, sheared)
    for kw in (dict(a=0.0, b=1.0), dict(a=0.5, b=0.3, x1=2, c1=0.7), dict(a=0.5, b=0.3, x1=2, c1=0.7, x2=3, c2=-0.2)):
        _close(*_both(s, 1, 0, **kw), s)
    _close(*_both(s, 1, 2, a=0.5, b=0.3, x1=2, c1=0.7, x2=2, c2=0.1), s)      # out is x1 and x2
    _close(*_both(s, 1, 1, a=1.0, b=0.3, x1=2, c1=0.7), s)                    # in place: face-value array


@pytest.mark.parametrize('kind', ['dgfs-wall-specular', 'dgfs-inlet', 'dgfs-inlet-normalshock', 'dgfs-outlet',
                                  'dgfs-vanish', 'dgfs-wall-diffuse-cyl', 'dgfs-wall-diffuse'])
@pytest.mark.parametrize('ndims,precision,Nv', [(2, 'single', 16), (3, 'single', 12), (2, 'double', 12), (3, 'double', 8)])
def test_affine_boundaries(cuda, kind, ndims, precision, Nv):
    names = ['x-', 'x+', 'y-', 'y+'] + (['z-', 'z+'] if ndims == 3 else [])
    s = _system(ndims, 2, Nv, precision, bcs={n: kind for n in names})
    _close(*_both(s, 1, 0, a=0.5, b=0.3, x1=2, c1=0.7, x2=3, c2=-0.2), s)
    _close(*_both(s, 1, 1, a=1.0, b=0.3), s)


@pytest.mark.parametrize('ndims,order,precision', [(2, 3, 'single'), (2, 2, 'double'), (3, 1, 'single'), (3, 2, 'single')])
def test_affine_unaligned_rows(cuda, ndims, order, precision):
    s = _system(ndims, order, 16, precision)
    want, _ = _both(s, 1, 0, a=0.5, b=0.3, x1=2, c1=0.7)
    for i in (0, 1, 2):
        b = s.eles_scal_upts_inb_full[i]
        n = torch.empty(b.numel() + 1, dtype=b.dtype, device=b.device)[1:].view(b.shape)
        s.eles_scal_upts_inb_full[i] = n.copy_(b)
    s.advect_combine(0.0, 1, 0, a=0.5, b=0.3, x1=2, c1=0.7)
    _close(s._bank(0).double(), want, s)


def test_affine_refuses(cuda):
    s = _system(2, 2, 16, 'single')
    L, r = _lib.lib(), _lib.ref
    u, o = s._bank(1), s._bank(0)
    call = lambda el, af, uf, out: L.bdgfs_fr_rhs_affine(r(el), r(s.walls.struct), r(af), u.data_ptr(), uf, out.data_ptr(),
                                                        0.0, 1.0, None, 0.0, None, 0.0, _lib.stream_ptr())
    assert call(s.ele.struct, s.ele.affine, None, o) == 0
    assert call(s.ele.struct, s.ele.affine, None, u) == -1                   # would read rows that it writes
    af = _lib.FrAffine.from_buffer_copy(s.ele.affine)
    af.p = 4
    assert call(s.ele.struct, af, None, o) == -3
    af.p, af.fid = 3, 0
    assert call(s.ele.struct, af, None, o) == -1

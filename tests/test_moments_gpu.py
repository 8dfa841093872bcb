"""bdgfs_moments / bdgfs_macroscopic against FP64 sums: every chunk width (8, 4
or 1 values of a z line), the smallest and odd grids, unaligned rows, both
precisions.

Tolerance: the sums have n = Nv^3 terms in FP64, so each raw moment is within
n eps of its sum of magnitudes (n eps <= 1.1e-11 at 37^3); q and P subtract
raw moments of their own size times |U|^2 <= 1 and |c|^2 <= 36."""
import numpy as np
import pytest
import torch

from oracle.fr import moments

pytestmark = pytest.mark.gpu


class Grid:
    def __init__(self, Nv, L=6.0):
        self.N, self.L = Nv, L

    def Nv(self): return self.N
    def vsize(self): return self.N**3
    def cw(self): return (2 * self.L / self.N)**3
    def c0(self): return np.linspace(-self.L + self.L / self.N, self.L - self.L / self.N, self.N)

    def cv(self):
        c = self.c0()
        return np.stack([a.ravel() for a in np.meshgrid(c, c, c, indexing='ij')])


def _rows(g, n, dtype):
    rng = np.random.default_rng(g.N)
    cv = g.cv()
    out = []
    for _ in range(n):
        u = rng.uniform(-0.5, 0.5, 3)[:, None]
        out.append(rng.uniform(0.5, 1.5) * np.exp(-np.sum((cv - u)**2, axis=0) / rng.uniform(0.7, 1.4))
                   * (1 + 0.1 * rng.uniform(-1, 1, cv.shape[1])))
    return torch.from_numpy(np.stack(out)).to(dtype).cuda()


@pytest.mark.parametrize('Nv', [1, 2, 7, 8, 12, 16, 20, 24, 32, 37])
@pytest.mark.parametrize('dtype', [torch.float32, torch.float64])
@pytest.mark.parametrize('shift', [0, 1])
def test_macroscopic_and_raw_moments(cuda, Nv, dtype, shift):
    from frfs_b200.system import macroscopic, raw_moments
    g = Grid(Nv)
    f = _rows(g, 3, dtype)
    buf = torch.empty(f.numel() + shift, dtype=dtype, device=f.device)
    f = buf[shift:].view(f.shape).copy_(f)
    raw = raw_moments(f, g).cpu().numpy()
    got = [a.cpu().numpy() for a in macroscopic(f, g)]
    cv, F = g.cv(), f.double().cpu().numpy()
    c2 = np.sum(cv * cv, axis=0)
    w = [np.ones_like(c2), *cv, cv[0]**2, cv[0] * cv[1], cv[0] * cv[2], cv[1]**2, cv[1] * cv[2], cv[2]**2,
         c2 * cv[0], c2 * cv[1], c2 * cv[2]]
    for i in range(3):
        for j in range(13):
            mag = np.sum(np.abs(w[j]) * F[i]) * g.cw()
            assert abs(raw[i, j] - np.sum(w[j] * F[i]) * g.cw()) <= 1e-11 * mag, (i, j)
        if Nv < 7:
            continue                       # no temperature on a grid this coarse
        want = moments(F[i], cv, g.cw())
        for a, b in zip(got, want):
            assert np.allclose(a[i], b, rtol=1e-11, atol=1e-10), (i, a[i], b)

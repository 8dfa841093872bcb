"""Indicator and projecting scatter with the row in shared memory against the
general streaming kernels (reached by the same rows one element off a 16-byte
boundary): every grid size that has that form and one that has none.

Both compute in FP64 from the same FP32 values, in different orders: 1e-13 of the
sums.  So FP32 outputs agree to one unit in the last place (1.2e-7) plus what the
deviation's cancellation lifts out of the sums (sur_s, eps: 1e-6), bf16 rows to one
bf16 unit (2^-7), and the lists hold the same rows."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(Nv, n, dev):
    rng = np.random.default_rng(Nv + n)
    c0 = (np.arange(Nv) + 0.5) * (12.0 / Nv) - 6.0
    x, y, z = np.meshgrid(c0, c0, c0, indexing='ij')
    out = []
    for i in range(n):
        u, T = rng.uniform(-0.4, 0.4, 3), rng.uniform(0.8, 1.3)
        m = np.exp(-((x - u[0])**2 + (y - u[1])**2 + (z - u[2])**2) / T)
        amp = 0.01 if i % 3 else 0.5
        out.append(rng.uniform(0.5, 2) * m * (1 + amp * np.sin(x + i) * np.cos(y - z)))
    f = torch.from_numpy(np.stack(out).reshape(n, -1)).float().to(dev)
    if n > 4:
        f[2] = 0.0                           # no density: to the spectral list
        f[4, 7] = float('nan')
    return c0, f


def _off(t):
    """The same values one element off a 16-byte boundary."""
    buf = torch.empty(t.numel() + 4, dtype=t.dtype, device=t.device)
    v = buf[1:1 + t.numel()].view(t.shape)
    v.copy_(t)
    return v


@pytest.mark.parametrize('Nv', [8, 16, 24, 32])
@pytest.mark.parametrize('n', [1, 9, 301])
def test_staged_rows(cuda, Nv, n):
    from frfs_b200 import _lib
    dev = torch.device('cuda')
    c0, f = _rows(Nv, n, dev)
    L, n3 = _lib.lib(), Nv**3
    c0d = torch.from_numpy(c0).to(dev)
    x = np.stack(np.meshgrid(c0, c0, c0, indexing='ij')).reshape(3, -1)
    phi = np.concatenate([np.ones((1, n3)), x, (x * x).sum(0)[None]])
    ginv = torch.from_numpy(np.linalg.inv(phi @ phi.T)).to(dev).contiguous()
    got = []
    for put in (lambda t: t, _off):
        i32 = lambda: torch.full((n,), -1, dtype=torch.int32, device=dev)
        flt = lambda *s: torch.zeros(*s, device=dev)
        b = dict(counts=torch.zeros(4, dtype=torch.int64, device=dev), sur=i32(), spec=i32(), fb=i32(),
                 inv=flt(n), rho2=flt(n), s=flt(n), eps=flt(n), uT=flt(n, 4),
                 flag=torch.zeros(n, dtype=torch.uint8, device=dev),
                 err=torch.zeros(2, dtype=torch.float64, device=dev),
                 dev=torch.zeros(n, n3, dtype=torch.bfloat16, device=dev))
        h = _lib.HybridArgs(
            ndof=n, Nv=Nv, fp64=0, c0=c0d.data_ptr(), ginv=ginv.data_ptr(), cw=(12.0 / Nv)**3, threshold=0.1,
            recheck=0.3, seed=5, counts=b['counts'].data_ptr(), sur_idx=b['sur'].data_ptr(),
            sur_inv_rho=b['inv'].data_ptr(), sur_rho2=b['rho2'].data_ptr(), spec_idx=b['spec'].data_ptr(),
            flag=b['flag'].data_ptr(), eps=b['eps'].data_ptr(), recheck_err=b['err'].data_ptr(), seed_dev=0,
            dev_rows=b['dev'].data_ptr(), feat=0, feat_ld=0, sur_s=b['s'].data_ptr(), fb_idx=b['fb'].data_ptr(),
            sur_uT=b['uT'].data_ptr(), center=0)
        fp = put(f)
        _lib.check(L.bdgfs_hybrid_classify(C.byref(h), fp.data_ptr(), _lib.stream_ptr()), 'classify')
        cnt = b['counts'].tolist()
        order = b['sur'][:cnt[0]].long()
        # a compact Q per surrogate row: a function of the row, so that the order
        # of the list does not matter; one row not finite
        Qc = (f[order] * torch.sin(torch.arange(n3, device=dev) * 0.37)).contiguous()
        if n > 4:
            Qc[order == 7, 11] = float('inf')
        Qc, Q = put(Qc), put(f * 0.5)
        if cnt[0]:
            _lib.check(L.bdgfs_hybrid_project_scatter(C.byref(h), Qc.data_ptr(), Q.data_ptr(), _lib.stream_ptr()),
                       'project_scatter')
        torch.cuda.synchronize()
        rows = {int(r): k for k, r in enumerate(order.tolist())}
        got.append((b, b['counts'].tolist(), rows, Q.clone()))
    (b, cnt, rows, Q), (w, wcnt, wrows, wQ) = got
    assert cnt == wcnt and set(rows) == set(wrows)
    assert set(b['spec'][:cnt[1]].tolist()) == set(w['spec'][:cnt[1]].tolist())
    assert b['fb'][:cnt[3]].tolist() == w['fb'][:cnt[3]].tolist()
    assert torch.equal(b['flag'], w['flag'])
    if n > 4:
        assert 0 < cnt[0] < n and {2, 4} <= set(b['spec'][:cnt[1]].tolist())
    close = lambda p, q, r: bool((abs(p - q) <= r * abs(q) + 1e-30).all())
    assert close(b['eps'], w['eps'], 1e-6)
    for r in rows:
        i, j = rows[r], wrows[r]
        for key in ('inv', 'rho2', 's'):
            assert close(b[key][i], w[key][j], 1e-6)
        assert float((b['uT'][i] - w['uT'][j]).abs().max()) < 1e-6
        p, q = b['dev'][i].float(), w['dev'][j].float()
        assert bool(((p - q).abs() <= q.abs() / 128 + 1e-9).all())
    fin = torch.isfinite(wQ)
    assert torch.equal(torch.isfinite(Q), fin)
    assert float((Q - wQ)[fin].abs().max()) <= 2.4e-7 * float(wQ[fin].abs().max())
    assert torch.allclose(b['err'], w['err'], rtol=1e-5, atol=0)

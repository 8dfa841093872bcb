"""The relaxation kernels' routes agree: 512 threads per row (few rows), 256
threads (many rows), and rows without 16-byte alignment (one value per step,
stage or order read from the arguments).  The 512-thread route is pinned to the
reference's kernels and the oracle elsewhere.

Few and many rows give the same bits.  Rows without alignment run the same FP64
arithmetic with the row sums added in another order: n eps = 3e-12 of the sums'
magnitudes (n = 24^3), which reach f through the targets; in FP32 the results round to neighbours at most (2^-23 each way,
with dt nu < 1 no amplification): 3e-7."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(name, Nv, dtype):
    from frfs_b200.adgfs import ADGFSScatteringModel
    from frfs_b200.backend import CUDABackend
    from frfs_b200.util import subclass_where
    from frfs_b200.velocitymesh import DGFSVelocityMesh
    from helpers import vhs_cfg
    cfg = vhs_cfg(Nv, 4, 6, 5, precision='double' if dtype == torch.float64 else 'single',
                  extra='muRef = 2.117e-5')
    cfg.set('scattering-model', 'type', name)
    be = CUDABackend(cfg)
    vm = DGFSVelocityMesh(be, cfg)
    return vm, subclass_where(ADGFSScatteringModel, scattering_model=name)(be, cfg, vm)


def _rows(vm, nbank, nrow, dtype):
    rng = np.random.default_rng(vm.Nv())
    cv = vm.cv()

    def one():
        u = rng.uniform(-0.3, 0.3, 3)[:, None]
        T = rng.uniform(0.8, 1.2)
        return rng.uniform(0.8, 1.2) / (np.pi * T)**1.5 * np.exp(-np.sum((cv - u)**2, axis=0) / T)
    return [torch.from_numpy(np.stack([one() for _ in range(nrow)])).to(dtype).cuda() for _ in range(nbank)]


def _place(rows, n, shift):
    """The rows repeated to n, at an offset of ``shift`` values."""
    x = rows[torch.arange(n) % rows.shape[0]]
    buf = torch.empty(x.numel() + shift, dtype=x.dtype, device=x.device)
    return buf[shift:].view(x.shape).copy_(x)


ROUTES = [(5, 0), (600, 0), (5, 1), (600, 1)]


def _agree(outs, dtype):
    tol = 3e-7 if dtype == torch.float32 else 1e-11
    for o in outs[1:]:
        assert float((o - outs[0]).abs().max() / outs[0].abs().max()) <= tol


@pytest.mark.parametrize('name', ['bgk-direct-gll', 'esbgk-direct-gll', 'shakov-direct-gll'])
@pytest.mark.parametrize('Nv,dtype', [(24, torch.float32), (16, torch.float64), (10, torch.float32), (4, torch.float64)])
def test_ars_and_bdf_routes(cuda, name, Nv, dtype):
    from frfs_b200.integrators import STEPPERS
    vm, sm = _model(name, Nv, dtype)
    f = _rows(vm, 4, 5, dtype)
    L = [0.2 * (a - b) for a, b in zip(f, f[1:] + f[:1])]
    A = STEPPERS['adgfs-ars-443']
    dt = 0.01
    per_stage = [[] for _ in range(4)]
    per_q = {2: [], 3: []}
    for n, shift in ROUTES:
        F, Ls = [_place(x, n, shift) for x in f], [_place(x, n, shift) for x in L]
        mom = lambda: torch.zeros(n, sm.nalph, dtype=torch.float64, device='cuda')
        U, LU = [mom() for _ in range(5)], [mom() for _ in range(4)]
        for ar in (1, 2, 3, 4):
            out = F[0] if ar == 4 else torch.empty_like(F[0])      # the last stage works in place
            sm.ars_stage(n, dt, ar, 2 | 4 | 8 | (1 if ar == 1 else 0), A._A_expl(ar), A._A_impl(ar), F[:ar], out,
                         Ls[:ar], U[:ar + 1], LU[:ar])
            per_stage[ar - 1].append(torch.cat([out[:5].double().flatten(), U[ar][:5].flatten()]))
        for q in (2, 3):
            B = STEPPERS[f'adgfs-bdf-{q}']
            Fq, Uq, LUq = [_place(x, n, shift) for x in f[:q]], [mom() for _ in range(q)], [mom() for _ in range(q)]
            for i in range(q - 1):
                sm.bdf_step(n, dt, 1, 1, [0.0, 1.0], [0.0], 0.0, [Fq[i]], Fq[i], [Ls[i]], [Uq[i]], [LUq[i]], mom())
            new = mom()
            sm.bdf_step(n, dt, q, 7, B.bdf_A, [-x for x in B.bdf_G], B.bdf_B, Fq, Fq[0], Ls[:q], Uq, LUq, new)
            per_q[q].append(torch.cat([Fq[0][:5].double().flatten(), new[:5].flatten()]))
    for outs in per_stage + list(per_q.values()):
        _agree(outs, dtype)


@pytest.mark.parametrize('name', ['bgk-direct-gll', 'esbgk-direct-gll', 'shakov-direct-gll'])
@pytest.mark.parametrize('Nv,dtype', [(24, torch.float32), (16, torch.float64), (10, torch.float32)])
def test_row_count_does_not_change_a_bit(cuda, name, Nv, dtype):
    """A row's moments, stage and BDF step have the same bits in a list of any
    length (a partitioned run is the serial one): every thread count of the
    kernels."""
    from frfs_b200.integrators import STEPPERS
    vm, sm = _model(name, Nv, dtype)
    f = _rows(vm, 3, 5, dtype)
    L = [0.2 * (a - b) for a, b in zip(f, f[1:] + f[:1])]
    A, B = STEPPERS['adgfs-ars-443'], STEPPERS['adgfs-bdf-2']
    outs = []
    for n in (5, 591, 592, 1500):
        F, Ls = [_place(x, n, 0) for x in f], [_place(x, n, 0) for x in L]
        mom = lambda: torch.zeros(n, sm.nalph, dtype=torch.float64, device='cuda')
        U, LU = [mom() for _ in range(4)], [mom() for _ in range(3)]
        got = []
        for ar in (1, 2, 3):
            out = torch.empty_like(F[0])
            sm.ars_stage(n, 0.01, ar, 2 | 4 | 8 | (1 if ar == 1 else 0), A._A_expl(ar), A._A_impl(ar), F[:ar], out,
                         Ls[:ar], U[:ar + 1], LU[:ar])
            got.append(out)
        Uq, LUq, new = [mom() for _ in range(2)], [mom() for _ in range(2)], mom()
        sm.bdf_step(n, 0.01, 1, 1, [0.0, 1.0], [0.0], 0.0, [F[0]], F[0], [Ls[0]], [Uq[0]], [LUq[0]], mom())
        out = torch.empty_like(F[0])
        sm.bdf_step(n, 0.01, 2, 7, B.bdf_A, [-x for x in B.bdf_G], B.bdf_B, F[:2], out, Ls[:2], Uq, LUq, new)
        outs.append([x[:5].clone() for x in got + [out, new] + U + LU + Uq + LUq])
    for o in outs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(o, outs[0]))

"""The single-RHS solver with its sums in the hop epilogues: half volumes below
a block (16), of ragged blocks (720), with the sums finished in the last block
(up to 512 blocks) and in a kernel of their own (576 blocks), in every sloppy
format; against the oracle's solution and its operator."""
import numpy as np
import pytest

import plqcd_b200 as P
from oracle import oracle as O
from tests.gpu_util import dev_bytes, field_from_host, field_to_host, new_lattice, to_dev

pytestmark = pytest.mark.gpu

SLOPPY = [(P.F64, 18), (P.F32, 18), (P.F32, 12), (P.F16, 12), (P.BF16, 12)]
KAPPA = 0.12


def _system(dims, seed=3):
    rng = np.random.default_rng(seed)
    V = O.volume(dims)
    u, b = O.random_su3(4 * V, rng).reshape(4 * V, 9), O.gaussian_spinor(V, rng)
    lat = new_lattice(dims)
    g = P.Gauge(lat, P.F64, 18)
    g.load_device(to_dev(u))
    return lat, g, u, b


def _solve(lat, g, b, prec, recon, **kw):
    gs = None
    if prec != P.F64:
        gs = P.Gauge(lat, prec, recon)
        gs.copy_from(g)
    be, bo = field_from_host(lat, b, 0, P.F64), field_from_host(lat, b, 1, P.F64)
    xe, xo = dev_bytes(lat.spinor_bytes(P.F64)), dev_bytes(lat.spinor_bytes(P.F64))
    raise_on_error = kw.pop("raise_on_error", True)
    info = P.invert_cg(lat, g, gs, xe, xo, be, bo, P.cg_param(kappa=KAPPA, tol=1e-10, sloppy_prec=prec, **kw),
                       raise_on_error=raise_on_error)
    return info, field_to_host(lat, xe, P.F64, 0) + field_to_host(lat, xo, P.F64, 1)


def _residual(restatement, dims, u, x, b):
    r = b - restatement.wilson(dims, u, x, KAPPA)
    return np.linalg.norm(r) / np.linalg.norm(b)


@pytest.mark.parametrize("prec,recon", SLOPPY)
@pytest.mark.parametrize("dims", [(2, 2, 2, 4), (10, 6, 4, 6), (16, 16, 16, 18)])
def test_solution(cuda, restatement, dims, prec, recon):
    lat, g, u, b = _system(dims)
    info, x = _solve(lat, g, b, prec, recon)
    assert info.converged == 1 and info.schur_residual <= 1e-10
    # |b - D x| / |b| follows from the Schur residual: the odd equation is solved exactly
    assert _residual(restatement, dims, u, x, b) < 2e-10
    assert abs(info.true_residual - _residual(restatement, dims, u, x, b)) < 1e-12
    again, y = _solve(lat, g, b, prec, recon)
    assert np.array_equal(x, y) and again.iterations == info.iterations
    assert info.sloppy_hops >= 4 * info.iterations


@pytest.mark.parametrize("prec,recon", [(P.F64, 18), (P.F16, 12)])
@pytest.mark.parametrize("max_iter", [1, 2, 7])
def test_stops_at_max_iter(cuda, restatement, prec, recon, max_iter):
    """Nothing of an iteration queued ahead shows in a solve that stops early:
    more iterations come closer, and the count is exact."""
    dims = (4, 6, 8, 10)
    lat, g, u, b = _system(dims)
    info, x = _solve(lat, g, b, prec, recon, max_iter=max_iter, raise_on_error=False)
    assert info.converged == 0 and info.iterations == max_iter
    more, y = _solve(lat, g, b, prec, recon, max_iter=max_iter + 5, raise_on_error=False)
    assert more.iterations == max_iter + 5
    assert _residual(restatement, dims, u, y, b) < _residual(restatement, dims, u, x, b) < 1.0


def test_zero_source(cuda):
    dims = (4, 4, 4, 6)
    lat, g, u, b = _system(dims)
    for prec, recon in SLOPPY:
        info, x = _solve(lat, g, np.zeros_like(b), prec, recon)
        assert info.converged == 1 and info.iterations == 0 and not x.any()


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("prec,recon", [(P.F64, 18), (P.F32, 18), (P.F16, 12), (P.BF16, 12)])
@pytest.mark.parametrize("dims,nrhs", [((2, 2, 2, 4), 3), ((10, 6, 4, 6), 1), ((10, 6, 4, 6), 2), ((4, 6, 8, 10), 5)])
def test_batch_residuals(cuda, restatement, dims, nrhs, prec, recon, use_graph):
    """The batched solver's FP64 residuals come out of its hops (two RHS per
    block, an idle one for odd counts; one RHS alone takes separate passes):
    every solution and every reported residual against the oracle."""
    lat, g, u, _ = _system(dims)
    rng = np.random.default_rng(9)
    b = [O.gaussian_spinor(lat.V, rng) for _ in range(nrhs)]
    gs = None
    if prec != P.F64:
        gs = P.Gauge(lat, prec, recon)
        gs.copy_from(g)
    nb = lat.spinor_bytes(P.F64)
    be, bo, xe, xo = (dev_bytes(nrhs * nb) for _ in range(4))
    for r in range(nrhs):
        be[r * nb:(r + 1) * nb] = field_from_host(lat, b[r], 0, P.F64)
        bo[r * nb:(r + 1) * nb] = field_from_host(lat, b[r], 1, P.F64)
    item = {"lat": lat, "g64": g, "g_sloppy": gs, "nrhs": nrhs, "x_even": xe, "x_odd": xo, "b_even": be, "b_odd": bo}
    info, res = P.invert_cg_batch([item], P.cg_param(kappa=KAPPA, tol=1e-10, sloppy_prec=prec), use_graph=use_graph)
    assert info.converged == 1 and info.max_schur_residual <= 1e-10
    for r in range(nrhs):
        x = field_to_host(lat, xe[r * nb:(r + 1) * nb], P.F64, 0) + field_to_host(lat, xo[r * nb:(r + 1) * nb], P.F64, 1)
        want = _residual(restatement, dims, u, x, b[r])
        assert want < 2e-10 and abs(res[r] - want) < 1e-12

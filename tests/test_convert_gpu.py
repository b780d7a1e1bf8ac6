"""The API-layout converters (spinor import / export, link import) against the
documented layouts, at volumes that leave part blocks and blocks across the
parities."""
import numpy as np
import pytest

import plqcd_b200 as P
from tests.gpu_util import new_lattice, torch

pytestmark = pytest.mark.gpu

# half volumes 16 (less than a warp), 72, 128 (one block), 420 and 960
DIMS = [(2, 4, 2, 2), (2, 2, 6, 6), (4, 4, 4, 4), (6, 10, 2, 14), (4, 6, 8, 10)]


def _random(shape):
    rng = np.random.default_rng(7)
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _planes(v, prec):
    """(Vh, 12) complex128 -> the stored numbers of one parity, as float64 (16-bit formats: values, norms)."""
    r = np.ascontiguousarray(v).view(np.float64).reshape(len(v), 24)
    if prec == P.F64:
        return r.reshape(-1, 12, 2).transpose(1, 0, 2), None
    r = r.astype(np.float32).astype(np.float64)
    if prec == P.F32:
        return r.reshape(-1, 6, 4).transpose(1, 0, 2), None
    m = np.abs(r).max(1)
    return (r / m[:, None]).reshape(-1, 3, 8).transpose(1, 0, 2), m


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("prec", [P.F64, P.F32, P.F16, P.BF16])
def test_spinor_import_export(cuda, dims, prec):
    t = torch()
    lat = new_lattice(dims)
    q = _random((lat.V, 12))
    q_dev = t.from_numpy(q).cuda()
    back = t.zeros_like(q_dev)
    for parity in (0, 1):
        f = t.zeros(lat.spinor_bytes(prec), dtype=t.uint8, device="cuda")
        lat.spinor_import(q_dev, parity, f, prec)
        lat.spinor_export(f, prec, parity, back)
        lat.synchronize()
        want, norms = _planes(q[parity * lat.Vh:(parity + 1) * lat.Vh], prec)
        if norms is None:
            got = f.view(t.float64 if prec == P.F64 else t.float32).cpu().numpy().reshape(want.shape)
            assert np.array_equal(got.astype(np.float64), want)
        else:
            kind = t.float16 if prec == P.F16 else t.bfloat16
            got = f[:48 * lat.Vh].view(kind).float().cpu().numpy().reshape(want.shape)
            assert np.array_equal(f[48 * lat.Vh:].view(t.float32).cpu().numpy(), norms.astype(np.float32))
            # half a unit in the last place of a value <= 1, and the FP32 rounding of 1 / norm and the product
            half_ulp = 2.0 ** -12 if prec == P.F16 else 2.0 ** -9
            assert np.abs(got - want).max() <= half_ulp + 2.0 ** -22
    tol = {P.F64: 0.0, P.F32: 2.0 ** -24, P.F16: 2.0 ** -11, P.BF16: 2.0 ** -8}[prec]
    scale = np.abs(q.view(np.float64)).max()
    assert np.abs((back.cpu().numpy() - q).view(np.float64)).max() <= tol * scale


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("prec,recon", [(P.F64, 18), (P.F64, 12), (P.F32, 18), (P.F32, 12), (P.F16, 12), (P.BF16, 12)])
def test_link_import(cuda, dims, prec, recon):
    t = torch()
    lat = new_lattice(dims)
    u = _random((2, lat.Vh, 4, 9))
    u /= np.abs(u).max()
    g = P.Gauge(lat, prec, recon)
    g.load_device(t.from_numpy(u).cuda())
    h = P.Gauge(lat, prec, recon)
    h.load_host(np.ascontiguousarray(u.reshape(4 * lat.V, 9)))
    lat.synchronize()
    assert np.array_equal(g.store_host(), h.store_host())
    stored = 9 if recon == 18 else 6  # row 2 of 12-real links is rebuilt for unitary links only
    got = g.store_host().reshape(2, lat.Vh, 4, 9)[..., :stored]
    want = u[..., :stored]
    if prec in (P.F16, P.BF16):  # the 16-bit formats round the FP32 value
        want = want.astype(np.complex64).astype(np.complex128)
    tol = {P.F64: 0.0, P.F32: 2.0 ** -24, P.F16: 2.0 ** -12, P.BF16: 2.0 ** -9}[prec]
    assert np.abs((got - want).copy().view(np.float64)).max() <= tol

"""The kernels that load the next directions into registers: the same bits as
the cp.async pipeline kernel (whose results the oracle tests check) in every
format and mode, at half volumes below a block, ragged in the last block, with
odd half extents, and over site ranges; FP64 also against the oracle."""
import numpy as np
import pytest

import plqcd_b200 as P
from oracle import oracle as O
from tests.gpu_util import dev_bytes, field_from_host, field_to_host, new_lattice, relmax, to_dev

pytestmark = pytest.mark.gpu

FORMATS = [(P.F64, 18), (P.F64, 12), (P.F32, 18), (P.F32, 12), (P.F16, 12), (P.BF16, 12)]
# half volumes 8 (a quarter of a warp), 120, 420 and 1440 (blocks of 64 and of 32 sites ragged or not)
DIMS = [(2, 2, 2, 2), (10, 6, 2, 2), (6, 10, 14, 2), (12, 4, 6, 10)]


# (variant, block): depth 1, depth 2, joined parities (full-lattice FP64)
CONFIGS = [(0, 64), (0, 128), (21, 64)]


def _force(monkeypatch, variant, block):
    monkeypatch.setenv("PLQCD_DSLASH_STAGES", str(variant))
    monkeypatch.setenv("PLQCD_DSLASH_BLOCK", str(block))


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("prec,recon", FORMATS)
def test_ahead_same_bits(cuda, monkeypatch, dims, prec, recon):
    lat = new_lattice(dims)
    g = P.Gauge(lat, prec, recon)
    g.random(11)
    nb = lat.spinor_bytes(prec)
    n = 3  # right-hand sides of the folded launch
    fe, fo, x = dev_bytes(n * nb), dev_bytes(n * nb), dev_bytes(n * nb)
    for r in range(n):
        lat.spinor_gaussian(fe[r * nb:], prec, 0, 20 + r)
        lat.spinor_gaussian(fo[r * nb:], prec, 1, 30 + r)
        lat.spinor_gaussian(x[r * nb:], prec, 0, 40 + r)
    flags = P.DSLASH_G5_IN | P.DSLASH_G5_OUT
    first, count = lat.Vh // 3, lat.Vh - lat.Vh // 3 - 1
    got = {}
    for v in [(2, 64)] + CONFIGS:
        _force(monkeypatch, *v)
        o = [dev_bytes(nb).fill_(7) for _ in range(5)]
        lat.dslash(g, o[0], fe, 1, prec)
        lat.dslash_xpay(g, o[1], fo, 0, prec, 0.25, x, -2.0, flags)
        lat.dslash_full(g, o[2], o[3], fe, fo, prec)
        lat.dslash_sites(g, o[4], fo, 0, prec, first, count, flags, 0.5, x, 1.5)
        monkeypatch.setenv("PLQCD_MRHS_VARIANT", str(100 + v[0]))
        monkeypatch.setenv("PLQCD_MRHS_BLOCK", str(v[1]))
        o.append(dev_bytes(n * nb))
        lat.dslash_mrhs_xpay(g, o[5], fo, n, 0, prec, 0.25, x, -2.0, flags)
        monkeypatch.delenv("PLQCD_MRHS_VARIANT")
        lat.synchronize()
        got[v] = o
    for v in CONFIGS:
        for k, (a, b) in enumerate(zip(got[v], got[2, 64])):
            assert bool((a == b).all()), (v, k)


@pytest.mark.parametrize("nrhs", [1, 2, 3, 5, 9])
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("prec,recon", FORMATS)
def test_multi_rhs_ahead_same_bits(cuda, monkeypatch, dims, prec, recon, nrhs):
    """The multi-RHS kernels that load ahead (RHS pairs; FP64 with the links
    of a block in shared memory, 2, 4 and 8 RHS per block, idle warps
    included) against the single-RHS pipeline kernel."""
    lat = new_lattice(dims)
    g = P.Gauge(lat, prec, recon)
    g.random(17)
    nb = lat.spinor_bytes(prec)
    f, x = dev_bytes(nrhs * nb), dev_bytes(nrhs * nb)
    for r in range(nrhs):
        lat.spinor_gaussian(f[r * nb:], prec, 1, 50 + r)
        lat.spinor_gaussian(x[r * nb:], prec, 0, 70 + r)
    flags = P.DSLASH_G5_IN | P.DSLASH_G5_OUT
    monkeypatch.setenv("PLQCD_MRHS_BLOCK", "64")
    got = {}
    for v in (102, *((4202, 4204, 4208) if prec == P.F64 else (2200, 2102))):
        monkeypatch.setenv("PLQCD_MRHS_VARIANT", str(v))
        o = [dev_bytes(nrhs * nb).fill_(7) for _ in range(2)]
        lat.dslash_mrhs(g, o[0], f, nrhs, 0, prec)
        lat.dslash_mrhs_xpay(g, o[1], f, nrhs, 0, prec, 0.25, x, -2.0, flags)
        lat.synchronize()
        got[v] = o
    for v, o in got.items():
        assert bool((o[0] == got[102][0]).all()) and bool((o[1] == got[102][1]).all()), v


@pytest.mark.parametrize("dims", DIMS[1:])
@pytest.mark.parametrize("config", [(0, 64), (21, 64)])
def test_ahead_f64_against_oracle(cuda, monkeypatch, restatement, dims, config):
    rng = np.random.default_rng(5)
    V = O.volume(dims)
    u, q = O.random_su3(4 * V, rng).reshape(4 * V, 9), O.gaussian_spinor(V, rng)
    lat = new_lattice(dims)
    g = P.Gauge(lat, P.F64, 18)
    g.load_device(to_dev(u))
    fe, fo = field_from_host(lat, q, 0, P.F64), field_from_host(lat, q, 1, P.F64)
    oe, oo = dev_bytes(lat.spinor_bytes(P.F64)), dev_bytes(lat.spinor_bytes(P.F64))
    _force(monkeypatch, *config)
    lat.dslash_full(g, oe, oo, fe, fo, P.F64)
    want = restatement.hop("eo", dims, q, u)
    want = restatement.hop("oe", dims, q, u, want)
    got = field_to_host(lat, oe, P.F64, 0) + field_to_host(lat, oo, P.F64, 1)
    assert relmax(got, want) < 1e-14


@pytest.mark.parametrize("prec,recon", [(P.F64, 18), (P.F32, 12), (P.F16, 12)])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (4, 6, 8, 10), (16, 16, 16, 32)])
def test_dependent_launches_back_to_back(cuda, monkeypatch, dims, prec, recon):
    """Launches that overlap their predecessor's end read all of its output
    and overwrite none of its input: a chain that hands two buffers back and
    forth gives the bits of the chain that waits after every launch."""
    lat = new_lattice(dims)
    g = P.Gauge(lat, prec, recon)
    g.random(3)
    nb = lat.spinor_bytes(prec)
    start = dev_bytes(nb)
    lat.spinor_gaussian(start, prec, 0, 8)
    _force(monkeypatch, 0, 64)
    got = []
    for wait in (True, False, False):
        a, b = start.clone(), dev_bytes(nb)
        for k in range(40):
            lat.dslash(g, b, a, 1, prec)
            if wait:
                lat.synchronize()
            lat.dslash_xpay(g, a, b, 0, prec, -0.01, a, 1.0)  # x is overwritten in place
            if wait:
                lat.synchronize()
        lat.synchronize()
        got.append(a)
    assert bool((got[0] == got[1]).all()) and bool((got[0] == got[2]).all())


@pytest.mark.parametrize("prec,recon", [(P.F64, 18), (P.F16, 12)])
@pytest.mark.parametrize("dims", [(4, 6, 8, 10), (16, 16, 16, 32)])
def test_overlapped_launch_waits_for_another_stream(cuda, monkeypatch, dims, prec, recon):
    """A launch that may overlap the one before it in its stream still waits
    for an event of another stream queued between the two: its input is
    written there, late, and overwritten once it has been read."""
    import torch
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    lat = P.Lattice(dims, 0, a.cuda_stream)
    g = P.Gauge(lat, prec, recon)
    g.random(3)
    nb = lat.spinor_bytes(prec)
    n = 12
    src, want, got = ([dev_bytes(nb) for _ in range(n)] for _ in range(3))
    inp, busy, other = (dev_bytes(nb) for _ in range(3))
    lat.spinor_gaussian(other, prec, 0, 7)
    _force(monkeypatch, 0, 64)
    for k in range(n):
        lat.spinor_gaussian(src[k], prec, 1, 100 + k)
        lat.dslash(g, want[k], src[k], 0, prec)
        got[k].fill_(7)
    torch.cuda.synchronize()
    for k in range(n):
        lat.dslash(g, busy, other, 1, prec)
        with torch.cuda.stream(b):
            torch.cuda._sleep(200000)  # (about 0.1 ms)
            inp.copy_(src[k])
            written = b.record_event()
        a.wait_event(written)
        lat.dslash(g, got[k], inp, 0, prec)
        b.wait_event(a.record_event())
    torch.cuda.synchronize()
    for k in range(n):
        assert bool((got[k] == want[k]).all()), k


@pytest.mark.parametrize("nrhs", [2, 3])
@pytest.mark.parametrize("prec,recon,variant", [(P.F64, 18, 4202), (P.F64, 12, 4204), (P.F32, 18, 2200),
                                                (P.F16, 12, 2200), (P.BF16, 12, 2200)])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (4, 6, 8, 10), (16, 16, 16, 16)])
def test_dependent_multi_rhs_launches_back_to_back(cuda, monkeypatch, dims, prec, recon, variant, nrhs):
    """The same chain with the multi-RHS kernels that overlap their predecessor."""
    lat = new_lattice(dims)
    g = P.Gauge(lat, prec, recon)
    g.random(3)
    nb = lat.spinor_bytes(prec)
    start = dev_bytes(nrhs * nb)
    for r in range(nrhs):
        lat.spinor_gaussian(start[r * nb:], prec, 0, 8 + r)
    monkeypatch.setenv("PLQCD_MRHS_VARIANT", str(variant))
    monkeypatch.setenv("PLQCD_MRHS_BLOCK", "64")
    got = []
    for wait in (True, False, False):
        a, b = start.clone(), dev_bytes(nrhs * nb)
        for k in range(40):
            lat.dslash_mrhs(g, b, a, nrhs, 1, prec)
            if wait:
                lat.synchronize()
            lat.dslash_mrhs_xpay(g, a, b, nrhs, 0, prec, -0.01, a, 1.0)  # x is overwritten in place
            if wait:
                lat.synchronize()
        lat.synchronize()
        got.append(a)
    assert bool((got[0] == got[1]).all()) and bool((got[0] == got[2]).all())


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("prec,recon", [(P.F32, 18), (P.F32, 12), (P.F16, 12), (P.BF16, 12)])
def test_packed_lanes_same_bits_as_scalar(cuda, monkeypatch, dims, prec, recon):
    """Packed FP32 lanes round as scalar FP32 does: the kernels that compute on
    them (two components of one site, or two right-hand sides) against the
    scalar arithmetic of the RHS-tile kernel."""
    lat = new_lattice(dims)
    g = P.Gauge(lat, prec, recon)
    g.random(13)
    nb = lat.spinor_bytes(prec)
    f, x = dev_bytes(2 * nb), dev_bytes(2 * nb)
    for r in range(2):
        lat.spinor_gaussian(f[r * nb:], prec, 1, 60 + r)
        lat.spinor_gaussian(x[r * nb:], prec, 0, 80 + r)
    flags = P.DSLASH_G5_IN | P.DSLASH_G5_OUT
    got = {}
    # 1: scalar, a thread per RHS; 100, 102, 103: the single-RHS kernels per RHS; 2200, 2102: RHS pairs
    for v, block in [(1, 64), (100, 64), (100, 128), (102, 64), (103, 64), (2200, 64), (2102, 64)]:
        monkeypatch.setenv("PLQCD_MRHS_VARIANT", str(v))
        monkeypatch.setenv("PLQCD_MRHS_BLOCK", str(block))
        o = [dev_bytes(2 * nb).fill_(7) for _ in range(2)]
        lat.dslash_mrhs(g, o[0], f, 2, 0, prec)
        lat.dslash_mrhs_xpay(g, o[1], f, 2, 0, prec, 0.25, x, -2.0, flags)
        lat.synchronize()
        got[v, block] = o
    for v, o in got.items():
        assert bool((o[0] == got[1, 64][0]).all()) and bool((o[1] == got[1, 64][1]).all()), v


@pytest.mark.parametrize("variant", [12, 13])
def test_two_site_numbers_refuse_what_they_refused(cuda, monkeypatch, variant):
    """12 and 13 stood for kernels of two sites per thread, which existed for
    one parity in 32 and 16 bits: there the numbers still run, elsewhere they
    are an error."""
    lat = new_lattice((4, 4, 4, 4))
    _force(monkeypatch, variant, 64)
    monkeypatch.setenv("PLQCD_MRHS_VARIANT", str(100 + variant))
    monkeypatch.setenv("PLQCD_MRHS_BLOCK", "64")
    for prec, recon in FORMATS:
        g = P.Gauge(lat, prec, recon)
        g.random(1)
        nb = lat.spinor_bytes(prec)
        a, b, c, d = (dev_bytes(nb) for _ in range(4))
        lat.spinor_gaussian(a, prec, 0, 2)
        lat.spinor_gaussian(b, prec, 1, 3)
        one = [lambda: lat.dslash(g, c, b, 0, prec), lambda: lat.dslash_xpay(g, c, b, 0, prec, 0.5, a, 1.0),
               lambda: lat.dslash_mrhs(g, c, b, 1, 0, prec)]
        refused = [lambda: lat.dslash_full(g, c, d, a, b, prec)]
        if prec == P.F64:
            refused += one + ([lambda: lat.dslash(g, c, b, 0, prec, P.DSLASH_COMPAT)] if recon == 18 else [])
        else:
            for call in one:
                call()
        for call in refused:
            with pytest.raises(P.PlqcdError, match="two sites per thread"):
                call()
    lat.synchronize()


@pytest.mark.parametrize("dims", DIMS)
def test_compat_configurations_same_bits(cuda, monkeypatch, dims):
    """Every configuration that the tuner tries for the bug-compatible hop."""
    lat = new_lattice(dims)
    g = P.Gauge(lat, P.F64, 18)
    g.random(19)
    nb = lat.spinor_bytes(P.F64)
    f = [dev_bytes(nb) for _ in range(2)]
    for par in (0, 1):
        lat.spinor_gaussian(f[par], P.F64, par, 90 + par)
    got = {}
    for v in [(2, 64), (2, 128), (2, 256), (0, 64), (0, 128), (0, 256), (3, 64), (3, 128)]:
        _force(monkeypatch, *v)
        got[v] = [dev_bytes(nb).fill_(7) for _ in range(2)]
        for par in (0, 1):
            lat.dslash(g, got[v][par], f[1 - par], par, P.F64, P.DSLASH_COMPAT)
        lat.synchronize()
    for v, o in got.items():
        assert bool((o[0] == got[2, 64][0]).all()) and bool((o[1] == got[2, 64][1]).all()), v

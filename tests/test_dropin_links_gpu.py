"""Which device copy of the links a host entry point uses. Each family keeps
one copy for its 18-real and one for its _short names; plqcd_gauge_update makes
both stale, and each stays so until its own upload."""
import ctypes
import os

import numpy as np
import pytest

import plqcd_b200 as P
from oracle import oracle as O
from tests.gpu_util import relmax

pytestmark = pytest.mark.gpu

L = (8, 4, 6, 4)


@pytest.fixture
def library(cuda):
    P.finalize_plqcd()
    path = O.write_input_file(L)
    assert P.init_plqcd(path) == 0, P.last_error()
    yield P.lib()
    P.finalize_plqcd()
    os.unlink(path)


def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


class _Split:
    names = ("single_mic_split_nohalfspinor", "single_mic_split_nohalfspinor_short")

    def __init__(self, q, u):
        self.q, self.u, self.out = P.aos_to_split(q), P.aos_to_split(u), P.aos_to_split(np.zeros_like(q))
        self.registered = self.u[0]

    def change(self, u):
        for old, new in zip(self.u, P.aos_to_split(u)):
            old[:] = new

    def call(self, name):
        f = getattr(P.lib(), "plqcd_hopping_matrix_eo_" + name)
        assert f(_ptr(self.out[0]), _ptr(self.out[1]), _ptr(self.u[0]), _ptr(self.u[1]), _ptr(self.q[0]), _ptr(self.q[1])) > 0
        out = np.zeros(self.out[0].shape, np.complex128)
        P.split_to_aos(self.out[0], self.out[1], out)
        return out


class _Packed:
    names = ("single_mic", "single_mic_short")

    def __init__(self, q, u):
        self.q, self.u = P.pack_lanes(q, 4), P.pack_lanes(u.reshape(-1, 36), 4)
        self.out = np.zeros_like(self.q)
        self.registered = self.u

    def change(self, u):
        self.u[:] = P.pack_lanes(u.reshape(-1, 36), 4)

    def call(self, name):
        assert getattr(P.lib(), "plqcd_hopping_matrix_eo_" + name)(_ptr(self.q), _ptr(self.out), _ptr(self.u)) > 0
        return P.unpack_lanes(self.out)


@pytest.mark.parametrize("first", [0, 1])
@pytest.mark.parametrize("family", [_Split, _Packed])
def test_links_changed_in_place_reach_both_copies(library, restatement, family, first):
    V = O.volume(L)
    rng = np.random.default_rng(41)
    q, u = O.gaussian_spinor(V, rng), O.random_su3(4 * V, rng)
    h = family(q, u)
    order = (h.names[first], h.names[1 - first])
    library.plqcd_gauge_update(h.registered.ctypes.data)
    for _ in range(3):
        want = restatement.hop("eo", L, q, u)[: V // 2]
        for name in order:  # (1e-13: the _short names rebuild row 2)
            assert relmax(h.call(name)[: V // 2], want) < 1e-13, name
        u = O.random_su3(4 * V, rng)
        h.change(u)
        library.plqcd_gauge_update(h.registered.ctypes.data)

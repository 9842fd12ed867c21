"""Branch-free arithmetic of csrc/it_math.h against the operation it stands for, bit for bit, on the CPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "irontimber_b200", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("math")
    src, so = d / "m.cpp", d / "m.so"
    src.write_text('#include "it_math.h"\n'
                   'extern "C" void quot(const float* a, const float* d, const float* r, int n, float* q, float* want, unsigned char* fits) {\n'
                   '  for (int i = 0; i < n; i++) { q[i] = it_quot(a[i], d[i], r[i]); want[i] = it_div(a[i], d[i]); fits[i] = it_quot_fits(a[i], d[i]); } }\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    return C.CDLL(str(so))


def quotients(lib, a, d, r):
    a, d, r = (np.ascontiguousarray(x, np.float32) for x in (a, d, r))
    q, want, fits = np.empty_like(a), np.empty_like(a), np.empty(a.size, np.uint8)
    p = lambda x: x.ctypes.data_as(C.c_void_p)
    lib.quot(p(a), p(d), p(r), a.size, p(q), p(want), p(fits))
    return q.view(np.uint32), want.view(np.uint32), fits.astype(bool)


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
def test_quotient_is_the_division(lib, ulps):
    """Reciprocals two units off either way (rcp.approx is within one); numerators and denominators at the edges of what is taken, signed zeros."""
    rng = np.random.default_rng(5 + ulps)
    n = 1 << 20
    a = np.concatenate([rng.standard_normal(n), rng.choice([-1, 1], n) * 10.0 ** rng.uniform(-14.9, 14.9, n)]).astype(np.float32)
    d = np.concatenate([1 + np.exp(-a[:n].astype(np.float64)), 10.0 ** rng.uniform(0, 14.9, n)]).astype(np.float32)
    up = lambda x: np.nextafter(np.float32(x), np.float32(np.inf))
    dn = lambda x: np.nextafter(np.float32(x), np.float32(0))
    ea = np.array([0.0, 1e-15, up(1e-15), dn(1e15), 1e15, 1.0, dn(1.0), up(1.0), 3.0, np.inf, 1e-40, np.nan], np.float32)
    ed = np.array([1.0, up(1.0), dn(2.0), 2.0, up(2.0), dn(1e15), 1e15, np.inf, 3.0, np.nan, dn(4.0)], np.float32)
    x, y = (g.ravel() for g in np.meshgrid(np.concatenate([ea, -ea]), ed))
    a, d = np.concatenate([a, x]), np.concatenate([d, y])
    with np.errstate(all="ignore"):
        r = (1.0 / d.astype(np.float64)).astype(np.float32)
    r = (r.view(np.int32) + np.int32(ulps)).view(np.float32)
    q, want, fits = quotients(lib, a, d, r)
    assert np.array_equal(q[fits], want[fits])
    assert fits[: 2 * n].mean() > 0.99
    edge = fits[2 * n:].reshape(ed.size, -1)
    assert edge[0, 0] and edge[0, ea.size] and not edge[0, 1] and edge[0, 2] and edge[0, 3] and not edge[0, 4]      # both zeros are taken, 1e-15 and 1e15 are not
    assert not edge[2].any() and not edge[6].any() and not edge[7].any() and not edge[9].any() and not edge[10].any()

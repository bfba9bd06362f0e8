"""The integer face fluxes of native FP64 (ptd_intflux.cuh): against exact
rational arithmetic on the CPU, and the GPU iteration on rough fields (wide
exponents, zeros, negative values) against the CPU oracle."""
import ctypes
import math
import os
import random
import struct
import subprocess
from fractions import Fraction

import numpy as np
import pytest

import ptdiff
from oracle import oracle as O
from ptdiff import scripts as S

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(ptdiff.__file__))), "csrc")
SOURCE = """
#include "ptd_intflux.cuh"
extern "C" int flux(int m, uint64_t a, uint64_t b, uint64_t c, uint64_t d, uint64_t* r)
{
    if (m == 0) return ptd::if_flux_lin(a, b, *r);
    if (m == 1) return ptd::if_flux_step(a, b, c, d, *r);
    return ptd::if_flux_cube(a, b, *r);
}
"""


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def value(b):
    return struct.unpack("<d", struct.pack("<Q", b))[0]


@pytest.fixture(scope="module")
def flux(tmp_path_factory):
    d = tmp_path_factory.mktemp("intflux")
    (d / "f.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "f.so"), str(d / "f.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "f.so"))
    lib.flux.argtypes = [ctypes.c_int] + [ctypes.c_uint64] * 4 + [ctypes.POINTER(ctypes.c_uint64)]

    def call(m, hl, hr, dl=1.0, dr=1.0):
        r = ctypes.c_uint64(0)
        return value(r.value) if lib.flux(m, bits(hl), bits(hr), bits(dl), bits(dr), ctypes.byref(r)) else None

    return call


def exact(m, hl, hr, dl=1.0, dr=1.0):
    hl, hr = Fraction(hl), Fraction(hr)
    return (1, Fraction(dl) + Fraction(dr), (hl + hr) ** 3)[m] * (hr - hl)


def pairs(n):
    rng = random.Random(3)
    ends = [0, 1, 2, 1 << 51, (1 << 52) - 2, (1 << 52) - 1]   # significands at the ends of a binade
    for k in range(n):
        if k % 3 == 0:
            x = value(bits(1.0) + rng.choice(ends))
            yield x, value(bits(1.0) + rng.choice(ends)) * 2.0 ** rng.randint(-31, 0)
        else:
            x = rng.uniform(1, 2) * 2.0 ** rng.randint(-199, 199)
            yield x, x * rng.choice([1.0, 1 + rng.uniform(-1e-14, 1e-14), 1 + rng.uniform(-1e-6, 1e-6),
                                     rng.uniform(0.5, 2), 2.0 ** rng.uniform(-29, 29)])


@pytest.mark.parametrize("m", [0, 1, 2], ids=["lin", "step", "cube"])
def test_flux_is_within_0_6_ulp(flux, m):
    rng = random.Random(m)
    for hl, hr in pairs(4000):
        dl = rng.uniform(1, 2) * 2.0 ** rng.randint(-199, 199)
        dr = dl * rng.choice([1.0, 2.0 ** rng.uniform(-29, 29)])
        for a, b in ((hl, hr), (hr, hl)):
            got, want = flux(m, a, b, dl, dr), exact(m, a, b, dl, dr)
            assert got is not None
            if want == 0:
                assert got == 0.0 and math.copysign(1.0, got) == 1.0
            else:
                assert abs(Fraction(got) - want) <= Fraction(6, 10) * Fraction(math.ulp(abs(float(want))))


def test_difference_within_a_factor_two_is_exact(flux):
    rng = random.Random(5)
    for _ in range(5000):
        x = rng.uniform(1, 2)
        y = x * rng.uniform(0.5, 2)
        assert flux(0, x, y) == y - x


@pytest.mark.parametrize("m", [0, 1, 2], ids=["lin", "step", "cube"])
def test_operands_out_of_range_are_declined(flux, m):
    for bad in (0.0, -0.0, -1.0, 5e-324, 1e-310, 2.0 ** -231, 2.0 ** 241, 2.0 ** -33, math.inf, -math.inf, math.nan):
        assert flux(m, bad, 1.0) is None and flux(m, 1.0, bad) is None
        if m == 1:
            assert flux(m, 1.0, 1.5, bad, 1.0) is None and flux(m, 1.0, 1.5, 1.0, bad) is None


# c and e are FP32 (2 x 2^-23 relative each), so the change of H over a few
# iterations agrees with the oracle's to a few times that.  (D = H^3: one
# iteration from a positive field; on a rough one the next iterates grow
# without bound, and where H = 0 the oracle's own dtau is NaN.)
@pytest.mark.gpu
@pytest.mark.parametrize("name,shape", [("diff_1D_lin", (131,)), ("diff_1D_nonlin", (77,)), ("diff_2D_lin", (70, 41)),
                                        ("diff_2D_linstep", (65, 38)), ("diff_2D_nonlin", (97, 36)),
                                        ("diff_3D_lin_multixpu", (33, 17, 12)), ("diff_3D_linstep_multixpu", (35, 16, 9)),
                                        ("diff_3D_nonlin_multixpu", (34, 18, 11))])
def test_rough_fields_match_the_oracle(name, shape):
    s = S.SCRIPTS[name]
    rng = np.random.default_rng(4)
    D = None
    if s.model == S.NONLIN:
        H0, niter = np.asfortranarray(2.0 ** rng.uniform(-36, 0, shape)), 1
    else:
        H0, niter = 2.0 ** rng.uniform(-12, 2, shape), 3
        H0[rng.random(shape) < 0.05] = 0.0
        H0[rng.random(shape) < 0.3] *= -1.0
        H0[rng.random(shape) < 0.05] *= 1e-80
        H0[rng.random(shape) < 0.02] = 5e-324
        H0 = np.asfortranarray(H0)
    if s.model == S.LINSTEP:
        D = np.asfortranarray(2.0 ** rng.uniform(-20, 0, shape))
    with ptdiff.Solver(ptdiff.make_params(s, shape)) as sol:
        sol.set_state(H0, D)
        sol.iterate(niter)
        H = sol.get_state().reshape(shape, order="F")
    Hr = np.array(H0, order="F")
    q = [np.zeros_like(Hr) for _ in range(3)]
    O.iterate(s, Hr, H0.copy(order="F"), q, niter, D=D)
    assert np.linalg.norm(H - Hr) <= 2e-6 * np.linalg.norm(Hr - H0)

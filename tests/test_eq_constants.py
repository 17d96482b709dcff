"""The constants of the flux's interface equilibrium (csrc/eq_constants.hpp):
every density at a face carries the factor 72 cd k0 and every mass flux 24 cd k1
/ s, which are 1 but for the constants' rounding, in the same direction on every
face. In exact arithmetic on the host, and as the bias of the pressure that the
flux kernel gives a fluid at rest on the GPU."""

import ctypes
import os
import subprocess
from fractions import Fraction as Q

import numpy as np
import pytest

from conftest import REPO
from plfbs import capi, cases

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("eq") / "libeq.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(REPO, "3d-plfbs-gpu_b200", "csrc"),
                    os.path.join(HERE, "eq_constants_host.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def _factors(k0, k1, cd, gamma, s):
    k0, k1, cd, c = Q(k0), Q(k1), Q(cd), Q(3, 2) * Q(s) ** 2 / Q(gamma)
    return [abs(float(x - 1)) for x in (72 * cd * k0, 24 * cd * k1 / Q(s), 72 * cd / c)]


def test_fp64_factors(host):
    k = (ctypes.c_double * 3)()
    for gamma in [0.5, 1.0, 1.1, 1.2, 1.3, 1.4, 5 / 3, 2.0, 3.0] + list(np.linspace(0.31, 4.7, 97)):
        host.eq64(ctypes.c_double(gamma), k)
        e = _factors(*k, gamma, 1.0)
        # both within half the unit roundoff's reach of 1, the quadratic terms'
        # factor within the places looked at
        assert max(e[:2]) <= 0.55 * 2.0 ** -53, (gamma, e)
        assert e[2] <= 9 * 2.0 ** -52, (gamma, e)


def test_fp32_factors(host):
    k = (ctypes.c_float * 3)()
    for gamma in (1.0, 1.3, 1.4):
        for U in [0.02, 0.05, 0.07, 0.1, 0.3] + list(np.linspace(0.011, 0.29, 41)):
            host.eq32(ctypes.c_double(gamma), ctypes.c_double(U), k)
            e = _factors(*k, gamma, U)
            plain = np.float32([U ** 2 * 1.5 / gamma / 72])[0]
            c = 1.5 * U * U / gamma
            p = _factors(float(np.float32(1 / c)), float(np.float32(2 * gamma / U)), float(plain),
                         gamma, U)
            assert sum(x * x for x in e) <= sum(x * x for x in p) * (1 + 1e-6), (gamma, U, e, p)
            assert e[2] <= 3 * 2.0 ** -23, (gamma, U, e)


@pytest.mark.gpu
@pytest.mark.parametrize("gamma", [1.0, 1.3])
def test_pressure_of_a_fluid_at_rest_has_no_bias(plfbs_lib, gamma):
    """Uniform density r at rest: a face's momentum flux is r / 3. Over 200
    densities the roundings (below one unit roundoff each, a handful) average
    out to less than 0.25 of it; the constants add 72 cd k0 - 1 (at most 0.5) and
    1 / 3's own rounding (0.5, downward): in all less than 0.75."""
    pm = cases.uniform_box(4, 4, 4, patch_types=["wall"] * 6)
    c = cases.Case(mesh_dir="", X=4, Y=4, Z=4, dt=0.1, mach=0.05, reynolds=50.0, ref_length=4.0,
                   bcs=[cases.BC("wall", 1, 0, 0, 0, "dirichlet", "neumann")])
    ma = cases.mesh_arrays(pm, c.visc, gamma, c.fneq_min)
    rt, vt, val = cases.bc_arrays(ma, c)
    s = capi.Solver(ma, rt, vt, val,
                    dict(visc=c.visc, gamma=gamma, dt=c.dt, max_velocity=c.mach, channel_height=4.0,
                         lengths=(4.0, 4.0, 4.0), gradient_mode=capi.GRAD_LS))
    n = np.asarray(ma.face_normal).reshape(-1, 3)[:ma.n_internal]
    faces = np.flatnonzero(n[:, 0] == 1.0)
    off = []
    for r in np.random.default_rng(5).uniform(0.9, 1.1, 200):
        q = np.zeros((ma.total_cells, 4))
        q[:, 3] = r  # (u, v, w, rho)
        s.set_state(q)
        s.run_stages(1)
        f = s.face_flux().reshape(-1, 4)[faces, 0]
        off.append(float(Q(float(f[len(f) // 2])) * 3 / Q(float(r)) - 1) * 2.0 ** 53)
        np.testing.assert_array_equal(f, f[0])
    s.close()
    assert max(abs(x) for x in off) < 8.0
    assert abs(np.mean(off)) < 0.75, np.mean(off)

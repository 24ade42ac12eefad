"""The sweeps' branch-free arithmetic (OpsSpec in euler_math.cuh) and its
out-of-line IEEE path against the C restatement, strict flavour: the right-hand
side must agree bit for bit whichever of the two a cell or face takes. States
mix ordinary cells with operands next to and outside OpsSpec's range: velocities
of zero, minus zero and 1e-200, densities of all-ones significands and scaled by
1e-125 and 1e+125, and cells near vacuum whose faces take the positivity
fallback. Grids leave a remainder of every tile (16 x 8, 8 x 16, 128)."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from cfd_inwsl_b200 import zone
from tests.util import gpu_solver

pytestmark = pytest.mark.gpu
ORACLE = Path(__file__).resolve().parent.parent / "oracle"
IM = {"wcns5": 2, "wenoz": 3, "teno": 11, "congz": 8, "muscl": 15}


@pytest.fixture(scope="module", autouse=True)
def _oracle():
    from tests.conftest import gpu_available
    if not gpu_available():
        pytest.skip("no CUDA device")
    if not (ORACLE / "_ref" / "libcfd_oracle.so").exists():
        if not (shutil.which("make") and shutil.which("gcc")):
            pytest.skip("no compiler for the C restatement")
        subprocess.run(["make", "-C", str(ORACLE), "_ref/libcfd_oracle.so"], check=True, capture_output=True)


def state(n, kind, rng):
    nc = int(np.prod(n))
    dim = len(n)
    rho = rng.uniform(0.5, 2.0, nc)
    vel = [rng.uniform(-1, 1, nc) for _ in range(dim)]
    p = rng.uniform(0.5, 2.0, nc)
    if kind == "edges":
        rho[rng.random(nc) < 0.3] = np.nextafter(1.0, 0.0)
        rho[rng.random(nc) < 0.2] = np.nextafter(1.0, 2.0)
        for v in vel:
            for x in (0.0, -0.0, 1e-200):
                v[rng.random(nc) < 0.15] = x
    elif kind == "vacuum":
        hole = rng.random(nc) < 0.1
        rho[hole], p[hole] = 1e-4, 1e-6
    elif kind in ("small", "large"):
        s = 1e-125 if kind == "small" else 1e125
        rho, p = rho * s, p * s
    return zone.prim_to_cons(np.stack([rho, *vel, p], -1))


@pytest.mark.parametrize("kind", ["plain", "edges", "vacuum", "small", "large"])
@pytest.mark.parametrize("n,scheme,flux,wrap", [
    ((131,), "wcns5", 0, False), ((259,), "teno", 1, False), ((97,), "wenoz", 0, False),
    ((37, 21), "wcns5", 0, True), ((16, 8), "teno", 1, True), ((33, 50), "wenoz", 1, False),
    ((21, 37), "congz", 0, False), ((29, 19), "muscl", 1, True),
    ((18, 9, 17), "wcns5", 0, True), ((11, 20, 8), "teno", 1, True), ((9, 7, 13), "wenoz", 0, False)])
def test_rhs_bits_match_the_restatement(n, scheme, flux, wrap, kind):
    from oracle.refsolver import ORC_OUTLET, ORC_WRAP, OracleC
    rng = np.random.default_rng(len(n) * 100 + n[0])
    cons = state(n, kind, rng)
    L = 1.0
    s = gpu_solver(len(n), list(n), [0, L, 0, L, 0, L], im=IM[scheme], fm=flux, strict=True, periodic=wrap)
    o = OracleC(len(n), list(n), L / n[0], IM[scheme], flux, [[ORC_WRAP if wrap else ORC_OUTLET] * 2] * 3)
    s.set_cons(cons)
    with np.errstate(all="ignore"):
        want = o.rhs(cons)
    got = s.rhsSolve()
    s.close()
    np.testing.assert_array_equal(got, want)


SCALES = {"inside_large": 1e60, "outside_large": 1e65, "inside_small": 1e-120, "mixed_large": 1e65, "mixed_small": 1e-125}


def scaled_state(n, kind, rng):
    """Density and pressure scaled to both sides of the range's ends (2^200 is
    1.6e60, 2^-400 is 3.9e-121), whole or in one half of the cells along x, so
    that faces and cells of both paths meet. The measures' squares stay finite
    (WENO-Z with periodic sides: beside an outlet's equal ghosts a measure of
    zero under a large one overflows its weight in any arithmetic)."""
    cons = state(n, "plain", rng)
    s = np.full(n[::-1], SCALES[kind])
    if kind.startswith("mixed"):
        s[..., : n[0] // 2] = 1.0 if "large" in kind else 1e-118
    return cons * s.reshape(-1, 1)


@pytest.mark.parametrize("kind", list(SCALES))
@pytest.mark.parametrize("n,scheme,flux,wrap", [
    ((131,), "wcns5", 0, False), ((259,), "teno", 1, False), ((97,), "wenoz", 0, True),
    ((37, 21), "wcns5", 0, True), ((16, 8), "teno", 1, True), ((33, 50), "wenoz", 1, True),
    ((21, 37), "congz", 0, False), ((29, 19), "muscl", 1, True),
    ((18, 9, 17), "wcns5", 0, True), ((11, 20, 8), "teno", 1, True), ((9, 7, 13), "wenoz", 0, True)])
def test_scaled_states_are_finite_and_match(n, scheme, flux, wrap, kind):
    from oracle.refsolver import ORC_OUTLET, ORC_WRAP, OracleC
    cons = scaled_state(n, kind, np.random.default_rng(len(n) * 100 + n[0]))
    o = OracleC(len(n), list(n), 1.0 / n[0], IM[scheme], flux, [[ORC_WRAP if wrap else ORC_OUTLET] * 2] * 3)
    want = o.rhs(cons)
    assert np.isfinite(want).all()
    s = gpu_solver(len(n), list(n), [0, 1.0] * 3, im=IM[scheme], fm=flux, strict=True, periodic=wrap)
    s.set_cons(cons)
    got = s.rhsSolve()
    s.close()
    np.testing.assert_array_equal(got, want)

"""Device functions and internal entry points by themselves (tests/device_check.cu)."""

import subprocess
from pathlib import Path

import pytest

from conftest import pkg_module

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    """check(name, *arguments): the figures that device_check prints."""
    build = pkg_module("build")
    exe = tmp_path_factory.mktemp("device_check") / "device_check"
    subprocess.run([build._nvcc(), "-O3", "-std=c++17", *build.ARCH, "-I", str(build.CSRC), "-o", str(exe),
                    str(Path(__file__).with_name("device_check.cu")), str(build.build()),
                    "-Xlinker", "-rpath", "-Xlinker", str(build.BUILD)], check=True)

    def run(*args):
        res = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=300)
        assert res.returncode == 0, res.stdout + res.stderr
        return [float(x) for x in res.stdout.split()]

    return run


@pytest.mark.parametrize("n", [40, 256, 300])
@pytest.mark.parametrize("e", [-80, -70, -50, 50, 80])
def test_block_inverses_scale(check, n, e):
    """Pivots whose square leaves the exponent range: the inverses are those of the unscaled
    factors times a power of two."""
    differ, not_finite = check("block_inverse", n, e)
    assert differ == 0 and not_finite == 0


def test_table_sine_and_cosine(check):
    """The FP64 kernels' sine and cosine of k r.  Absolute: three roundings of 2^-54 and the
    polynomials' 1e-17, below 2e-16, with the host's table; where the CTA computes the table
    (sincospi, 2 units in the last place) 2^-52 takes the place of one of them.  Up to half a unit
    h of angle the sine is c0 x + c1 x^3 with c1 moved by 0.87 / 4 of h^5 / 120: relative error
    h^4 / 120 times max |x^4 - 0.2175 x^2| = 0.0118, 8.7e-15, and five roundings of 2^-53."""
    n, host_table, device_table, small = check("sincos")
    assert n > 100000
    assert host_table <= 2e-16
    assert device_table <= 2e-16 - 2.0**-54 + 2.0**-52
    assert small <= 8.8e-15 + 5 * 2.0**-53


def test_reported_launches(check):
    """stats["kernel_launches"] counts the right-hand side's and the regular pairs' launches by
    formula: they are those of the launches captured in a graph."""
    calls, wrong = check("launch_counts")
    assert calls == 2 * 64 * 5 and wrong == 0


@pytest.mark.parametrize("n,nrhs", [(33, 1), (256, 3), (300, 4), (1000, 2)])
def test_substitution_of_orders_that_the_block_solves_do_not_hold(check, n, nrhs):
    """The cluster substitution (mixed form, orders above 43,264) against the block solves.  Both
    are backward stable: ||P b - L U x|| <= 2 n 2^-24 (sqrt 8 for complex products) of
    || |L| |U| |x| ||, in practice far below; the difference is that times the condition of
    these well-conditioned triangles (below 100)."""
    diff, residual = check("solves", n, nrhs)
    bound = 2 * n * 2.0**-24 * 8**0.5
    assert residual <= bound and diff <= 100 * bound


@pytest.mark.parametrize("n,nrhs", [(300, 4), (520, 3), (9602, 4)])
def test_right_hand_sides_together_and_alone(check, n, nrhs):
    """A right-hand side's sums do not depend on how many share the factors' reads; at 9,602
    rows a cluster holds two of the four at a time."""
    differ, not_finite = check("rhs_groups", n, nrhs)
    assert differ == 0 and not_finite == 0


def test_edges_of_the_dispatch(check):
    assert check("edges") == [1, 0, 2, 1, 1, 0]

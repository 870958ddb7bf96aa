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

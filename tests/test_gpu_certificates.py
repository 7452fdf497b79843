"""The traversal step's shortcuts against the plain forms they stand for, in
the product's own device functions (tests/native/certificates.cu, compiled
here): wherever a shortcut calls its result certain, the plain form gives the
same bits.  A shortcut that certified nothing would pass that trivially and
cost the step its speed, so each has the least share of its cases it must
certify, from how its inputs are drawn:

* reciprocal, channels: all (every float of the range; a channel's two forms
  differ on midpoints of 28 equal bits only);
* planes: all but determinants that cancel to RDELTA and numerators that
  underflow, a few in 10^4;
* psi: all but 2^-12 to 2^-10 of the coordinates, twice per pair;
* zeta: half the pairs have sums below 16 of which 11 is the limit, the others
  any exponent;
* exits: one ray in four lies inside a random entry face, half of the rays lie
  close to an edge; lattice rays lie on one more often than not;
* extinctions: half the draws of the longest edge give a quotient below 1000.
"""
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

LEAST = {
    "reciprocal": 1.0, "planes": 0.999, "planes_scalar_2^-30": 0.99, "planes_scalar_2^-60": 0.99,
    "planes_scalar_2^-80": 0.95, "planes_scalar_2^-100": 0.0, "planes_scalar_2^-118": 0.0,
    "planes_scalar_2^-140": 0.0, "planes_constant_scalar": 0.0, "planes_constant_depth": 0.0,
    "psi": 0.996, "zeta": 0.5, "zeta_powers_of_two": 0.25, "exits": 0.1, "exits_lattice": 0.05,
    "exits_edge_on": 0.0, "extinctions": 0.4, "channels": 0.999,
}


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("cert") / "certificates")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-I", os.path.join(ROOT, "vfray_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "native", "certificates.cu"), "-o", exe],
                   check=True, timeout=600)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    rows = [line.split() for line in out.stdout.splitlines()]
    return {r[0]: tuple(int(x) for x in r[1:]) for r in rows}


@pytest.mark.parametrize("name", sorted(LEAST))
def test_certified_results_are_the_plain_ones(name, counts):
    cases, sure, bad = counts[name]
    assert bad == 0 and cases >= 1 << 20
    assert sure >= LEAST[name] * cases, (sure, cases)

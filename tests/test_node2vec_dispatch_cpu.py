"""The node2vec kernels count the edge set's sectors in 32 bits: a graph whose
sectors do not fit is the general kernels'.  The rule, asked on the host at the
sizes around the line (no graph of that size is made)."""

import os
import shutil
import subprocess

import pytest

from knightking_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))
TOP = 1 << 32


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    if shutil.which(build.nvcc()) is None:
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("rule") / "rule")
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS + [os.path.join(HERE, "node2vec_dispatch.cu"), "-o", exe],
                   check=True)

    def ask(cases):
        text = "".join("%d %d %d %d %d\n" % c for c in cases)
        lines = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
        assert len(lines) == len(cases)
        return [ln.split()[-1] == "yes" for ln in lines]

    return ask


def test_sectors_in_32_bits(rule):
    cases = []
    for shift in (0, 1, 2):
        for E in (0, 5, 28_000_000, 1 << 30, TOP - 1):
            edge = TOP - 1 - (E >> shift)  # the last V whose sectors, (E >> shift) + V + 1, are 2^32 or fewer
            cases += [(V, E, shift, 1, 1) for V in (1, edge - 1, edge, edge + 1, TOP - 1) if 0 < V < TOP]
    for (V, E, shift, _, _), yes in zip(cases, rule(cases)):
        assert yes == ((E >> shift) + V + 1 <= TOP), (V, E, shift)


def test_needs_edge_set_and_offsets(rule):
    assert rule([(100, 1000, 1, 1, 1), (100, 1000, 1, 0, 1), (100, 1000, 1, 1, 0)]) == [True, False, False]

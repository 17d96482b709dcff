"""Which meshes march (csrc/march_rules.hpp): the side of the line that was faster
for each measured mesh, from us per step of both ways on a B200."""

import ctypes
import os
import subprocess

import pytest

from conftest import REPO

HERE = os.path.dirname(os.path.abspath(__file__))
SMS = 148

# compact, fp32, tiles, faces of the largest, faces, march, graph
MEASURED = [
    # uniform boxes, tables in shared memory
    (1, 0, 144, 384, 43200, 31, 59), (1, 0, 146, 1216, 146109, 53.9, 75.9),
    (1, 1, 148, 2496, 320348, 61.0, 75.9),
    # boxes graded along one axis, tables in L2
    (1, 0, 125, 160, 13056, 26.1, 55.3), (1, 0, 147, 864, 101376, 51.2, 69.7),
    (1, 0, 141, 1504, 180000, 76.1, 81.9), (1, 1, 146, 2912, 313920, 73.1, 76.0),
    # a record per face: tetrahedra, boxes graded along three axes
    (0, 0, 94, 192, 12600, 27.3, 51.2), (0, 0, 143, 768, 84474, 52.4, 67.7),
    (0, 0, 125, 832, 75581, 52.3, 63.5), (0, 0, 128, 864, 88492, 52.6, 69.5),
    (0, 0, 145, 992, 113778, 63.7, 72.0), (0, 0, 143, 1152, 130680, 70.2, 75.8),
    (0, 0, 144, 1152, 142112, 66.5, 77.4),
    (0, 0, 137, 928, 71928, 69.0, 65.5), (0, 0, 135, 1248, 119969, 87.7, 73.8),
    (0, 0, 144, 1216, 142112, 83.4, 75.8), (0, 0, 141, 1472, 168180, 91.6, 82.0),
    (0, 0, 147, 1568, 201728, 97.1, 86.0),
    (0, 1, 137, 1088, 108644, 43.6, 55.3), (0, 1, 144, 1664, 199511, 56.3, 65.7),
    (0, 1, 144, 1760, 214968, 61.8, 71.1), (0, 1, 139, 1728, 177280, 54.6, 63.8),
    (0, 1, 137, 1216, 121340, 62.8, 57.3), (0, 1, 142, 1760, 182918, 76.7, 65.1),
    (0, 1, 148, 2240, 240570, 89.1, 75.9), (0, 1, 148, 2272, 277553, 107.1, 73.8),
]


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("march") / "librules.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(REPO, "3d-plfbs-gpu_b200", "csrc"),
                    os.path.join(HERE, "march_rules_host.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("compact,fp32,n,SF,F,march,graph", MEASURED)
def test_the_faster_way(rules, compact, fp32, n, SF, F, march, graph):
    takes = rules.march_may_win(compact, fp32, SMS, F) and rules.march_wins(compact, fp32, n, SF, F)
    assert bool(takes) == (march < graph)

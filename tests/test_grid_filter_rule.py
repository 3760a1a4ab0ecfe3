"""Which DEMs the FP64 grid search takes behind its FP32 filter (grid_filter_ok, kernels.hpp):
the filter's offsets are 32 bits, its heights FP32, its bounds need positive indices and evenly
spaced axes."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

# nx, ny, evenly spaced, n1, n2, lowest and highest height: filtered
CASES = [
    ((64, 64, 1, 1.0, 2.0, -1.0, 1.0), 1),
    ((2, 2, 1, 1.0, 2.0, 0.0, 0.0), 1),
    ((1, 64, 1, 1.0, 2.0, 0.0, 0.0), 0),
    ((64, 1, 1, 1.0, 2.0, 0.0, 0.0), 0),
    ((0, 0, 1, 1.0, 2.0, 0.0, 0.0), 0),
    ((64, 64, 0, 1.0, 2.0, 0.0, 0.0), 0),
    ((64, 64, 1, -1.0, 2.0, 0.0, 0.0), 0),
    ((64, 64, 1, 1.0, 0.0, 0.0, 0.0), 0),
    ((64, 64, 1, 1.0, 2.0, "-inf", 1.0), 0),        # a height of -1e39 in FP32
    ((64, 64, 1, 1.0, 2.0, 0.0, "inf"), 0),
    ((64, 64, 1, 1.0, 2.0, -3e38, 3e38), 1),
    ((65536, 32767, 1, 1.0, 2.0, 0.0, 0.0), 1),     # 2^31 - 65536 offsets
    ((65536, 32768, 1, 1.0, 2.0, 0.0, 0.0), 0),     # 2^31
    ((65533, 32768, 1, 1.0, 2.0, 0.0, 0.0), 0),     # 2^31 with the rows' padding
    ((1 << 20, 1 << 20, 1, 1.0, 2.0, 0.0, 0.0), 0),
]


@pytest.fixture(scope="module")
def answers(tmp_path_factory):
    exe = tmp_path_factory.mktemp("filter") / "grid_filter"
    subprocess.run(["/usr/bin/g++", "-O1", "-std=c++17", f"-I{ROOT / 'c-_bistatic_sar_b200' / 'csrc'}",
                    f"-I{ROOT / 'include'}", "-I/usr/local/cuda/include",
                    str(Path(__file__).parent / "compat" / "grid_filter_driver.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    text = "\n".join(" ".join(map(str, c)) for c, _ in CASES)
    return subprocess.run([str(exe)], input=text, check=True, capture_output=True, text=True).stdout.split()


@pytest.mark.parametrize("k", range(len(CASES)))
def test_rule(answers, k):
    assert int(answers[k]) == CASES[k][1]

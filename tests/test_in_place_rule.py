"""Device samples are read in place only where a kernel can: memory of the
handle's own GPU, aligned, the whole range inside one allocation."""
import subprocess

import pytest

from conftest import ROOT

BASE, SIZE, N = 0x7f0000000000, 1 << 20, 8 * 4096  # an allocation, bytes read


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    exe = tmp_path_factory.mktemp("rule") / "in_place_rule"
    subprocess.run(["g++", "-std=c++17", "-x", "c++", f"-I{ROOT / 'fdas_gb300' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "in_place_rule.cpp"), "-o", str(exe)], check=True)

    def ask(*row):
        r = subprocess.run([str(exe)], input=" ".join(map(str, row)), capture_output=True, text=True, check=True)
        return r.stdout.strip() == "1"

    return ask


@pytest.mark.parametrize("what,row,want", [
    ("own memory", (1, 0, BASE, SIZE, BASE, N, 8, 0), True),
    ("inside it", (1, 0, BASE, SIZE, BASE + 512, N, 8, 0), True),
    ("up to its end", (1, 1, BASE, SIZE, BASE + SIZE - N, N, 8, 1), True),
    ("another GPU's", (1, 1, BASE, SIZE, BASE, N, 8, 0), False),
    ("host, managed or unknown", (0, 0, BASE, SIZE, BASE, N, 8, 0), False),
    ("odd float", (1, 0, BASE, SIZE, BASE + 4, N, 8, 0), False),
    ("past the end", (1, 0, BASE, SIZE, BASE + SIZE - N + 8, N, 8, 0), False),
    ("longer than it", (1, 0, BASE, SIZE, BASE, SIZE + 8, 8, 0), False),
    ("before it", (1, 0, BASE, SIZE, BASE - 8, N, 8, 0), False),
    ("range unknown", (1, 0, 0, 0, BASE, N, 8, 0), False),
])
def test_in_place(rule, what, row, want):
    assert rule(*row) is want

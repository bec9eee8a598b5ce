"""The split of small products over CTAs is found without a scan of every count.

The allocation-free entry point plans in every call, so the search must cost
less than the 8 to 30 us of the kernel it plans."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    exe = tmp_path_factory.mktemp("split") / "split_probe"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{ROOT / 'rawspec_gb300' / 'csrc'}",
                    str(ROOT / "tests" / "probe" / "split_probe.cpp"), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True)


def test_split_is_that_of_every_count_at_a_few(probe):
    res = probe
    assert res.returncode == 0, res.stdout
    tried = [int(line.split()[1]) for line in res.stdout.splitlines() if line.startswith("tried")]
    assert len(tried) == 10 and max(tried) <= 300, res.stdout


def test_one_unit_is_not_split_beyond_what_its_sum_costs(probe):
    chunks = [line.split()[1:] for line in probe.stdout.splitlines() if line.startswith("chunks")]
    assert len(chunks) == 3 and all(int(c) <= 8 or finalize == "1" for c, finalize in chunks), probe.stdout


def test_large_spectra_are_not_split_over_a_pair(probe):
    pairs = [line.split()[1] for line in probe.stdout.splitlines() if line.startswith("pair")]
    assert pairs == ["1", "1"], probe.stdout

"""The split of small products over CTAs is found without a scan of every count.

The allocation-free entry point plans in every call, so the search must cost
less than the 8 to 30 us of the kernel it plans."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_split_is_that_of_every_count_at_a_few(tmp_path):
    exe = tmp_path / "split_probe"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{ROOT / 'rawspec_gb300' / 'csrc'}",
                    str(ROOT / "tests" / "probe" / "split_probe.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
    tried = [int(line.split()[1]) for line in res.stdout.splitlines() if line.startswith("tried")]
    assert len(tried) == 10 and max(tried) <= 300, res.stdout

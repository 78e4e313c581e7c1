"""The phased re-quantiser's threshold tables on the CPU (quant_table_check.cpp):
where they are used they decide as the nearest-level search does, for every sample."""
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_thresholds_decide_as_the_search(tmp_path):
    exe = tmp_path / "quant_table_check"
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I",
                    str(ROOT / "fx-corr_b200" / "csrc"), str(ROOT / "tests" / "quant_table_check.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    searched, compared, stepped, samples, differ = map(int, out.split())
    assert searched > 20 and compared > 20 and stepped > 20 and samples > 1_000_000
    assert differ == 0

"""The lane density pass takes one target per lane or pairs, whichever was the faster by 2 % or more at the
sizes where both were measured (4,864 resident warps, particles at the rest spacing; alone or overlapped
with other streams, and within the judge's steps)."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent
MEASURED = {(0, "one"): [40000, 80000, 110000, 130000],
            (0, "pairs"): [165000, 175000, 185000, 230000, 290000, 311000, 330000, 380000, 400000, 500000, 560000, 622000,
                           800000, 1048576],
            (1, "one"): [150000, 300000, 350000],
            (1, "pairs"): [180000, 200000, 230000, 420000, 520000, 700000]}


def test_rule_follows_the_measurements(tmp_path):
    exe = tmp_path / "lane_rule"
    subprocess.run(["g++", "-std=c++17", "-o", str(exe), str(HERE / "cpp" / "lane_rule.cpp")], check=True)
    for (judge, variant), sizes in MEASURED.items():
        args = [str(v) for n in sizes for v in (n, 4864, judge)]
        got = subprocess.run([str(exe), *args], capture_output=True, text=True, check=True).stdout.split()
        assert got == [variant] * len(sizes)

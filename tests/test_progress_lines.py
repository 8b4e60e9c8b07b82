"""sym_fold's progress lines on the CPU: one every 5 s, as the reference prints
them, and one as a count that printed any ends."""
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

MAIN = """
void count(double seconds, bool stream) {
    Progress p;
    ProgressPrinter printer(p, stream, 100);
    p.completed = 40;
    std::this_thread::sleep_for(std::chrono::duration<double>(seconds));
    p.completed = 100;
}
}  // namespace
int main() {
    std::thread other([] { count(10.6, true); });
    std::thread brief([] { count(0.2, false); });
    count(6.3, false);
    other.join();
    brief.join();
}
"""


def test_progress_lines_every_five_seconds(tmp_path):
    text = (ROOT / "map_folding_gb300" / "csrc" / "cli_sym_fold.cpp").read_text()
    (tmp_path / "p.cpp").write_text(text[:text.index("void usage(")] + MAIN)
    subprocess.run(["g++", "-std=c++17", "-w", "-I", str(ROOT / "include"), str(tmp_path / "p.cpp"), "-o",
                    str(tmp_path / "p"), "-pthread"], check=True)
    err = subprocess.run([str(tmp_path / "p")], check=True, capture_output=True, text=True).stderr
    runs = {False: re.findall(r"^progress=(\d+)/100 rate=\S+/s elapsed_s=(\S+)$", err, re.M),
            True: re.findall(r"^stream selected=0 completed=(\d+) .* elapsed_s=(\S+)$", err, re.M)}
    for stream, at in ((False, [5, 6.3]), (True, [5, 10, 10.6])):
        assert [float(s) for _, s in runs[stream]] == pytest.approx(at, abs=0.4), err
        assert [c for c, _ in runs[stream]] == ["40"] * (len(at) - 1) + ["100"], err

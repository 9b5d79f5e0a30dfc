"""The prefill kernel's product order on the CPU: every ring unit taken and released in order, every S buffer overwritten
only once the PV that read it was waited for, every barrier met in the right phase, no wait that nothing ends."""
import subprocess
from pathlib import Path


def test_every_hand_off_of_the_product_order(tmp_path):
    src = Path(__file__).resolve().parent / "prefill_schedule_check.cpp"
    exe = tmp_path / "check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wno-unknown-pragmas", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout

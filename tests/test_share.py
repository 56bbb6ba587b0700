"""CPU check of the hand-over of shared sightlines (fsg_share.cuh): threads in the
place of blocks under the thread sanitizer, which reports a load of the bound or
of the sums that the flags' loads do not order."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "fake_spectra_gb300", "csrc")


@pytest.mark.parametrize("threads,nlos,chunks", [(8, 1, 400), (8, 3, 200), (6, 40, 9), (3, 8, 1)])
def test_hand_over_is_ordered(tmp_path, threads, nlos, chunks):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    flags = [cc, "-O1", "-g", "-std=c++17", "-fsanitize=thread", "-pthread", "-x", "c++"]
    probe = tmp_path / "probe.cpp"
    probe.write_text("int main() { return 0; }\n")
    pexe = str(tmp_path / "probe")
    if subprocess.run(flags + ["-o", pexe, str(probe)], capture_output=True).returncode or \
            subprocess.run([pexe], capture_output=True).returncode:
        pytest.skip("no thread sanitizer")
    exe = str(tmp_path / "share")
    subprocess.run(flags + ["-I", CSRC, "-o", exe, os.path.join(HERE, "share.cpp")], check=True)
    for _ in range(5):
        out = subprocess.run([exe, str(threads), str(nlos), str(chunks)], capture_output=True,
                             text=True, timeout=120)
        assert out.returncode == 0, out.stderr[:4000]
        assert [float(v) for v in out.stdout.split()] == [chunks * (3.0 + q) for q in range(nlos)]

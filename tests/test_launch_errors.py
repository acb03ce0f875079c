"""A launch that fails is reported: a loop body captured without its plane R has
no loop test and would never end.  The folded launches are [[nodiscard]] and the
build turns a dropped result into an error; here the same on a two-line file."""
import os
import re
import subprocess

from conftest import ROOT

SOLVER = os.path.join(ROOT, "3d-rism-cuda_b200", "csrc", "solver.cu")


def test_folded_launches_return_their_error():
    with open(SOLVER) as f:
        text = f.read()
    for fn in ("launch_split", "launch_fused", "launch_iteration"):
        assert re.search(r"\[\[nodiscard\]\] cudaError_t %s\(" % fn, text), fn
        calls = re.findall(r"(?m)^\s*(?:else )?%s<[^;]*;" % fn, text)
        assert not calls, calls


def test_build_rejects_a_dropped_launch_error(tmp_path):
    from rism3d_b200 import build as B
    src = tmp_path / "drop.cu"
    src.write_text("[[nodiscard]] cudaError_t launch(int n) { return n ? cudaSuccess : cudaErrorUnknown; }\n"
                   "void run() { launch(1); }\n")
    cmd = [B.NVCC] + B._flags() + ["-c", str(src), "-o", str(tmp_path / "drop.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode != 0 and "unused" in r.stderr + r.stdout
    src.write_text(src.read_text().replace("{ launch(1); }", "{ cudaError_t e = launch(1); (void)e; }"))
    assert subprocess.run(cmd, capture_output=True).returncode == 0

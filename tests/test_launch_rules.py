"""Rules that choose a launch's shape, compiled from the library's own header and run on the host."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _run(tmp_path, body):
    cc = shutil.which("g++") or shutil.which("c++")
    if cc is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    src = tmp_path / "rule.cpp"
    src.write_text('#include <cstdio>\n#include "pcsf_internal.h"\nusing namespace pcsf;\nint main()\n{\n%s\n}\n' % body)
    exe = tmp_path / "rule"
    subprocess.run([cc, "-std=c++17", "-I", os.path.join(ROOT, "phylocsf_gb300", "csrc"), "-I",
                    os.path.join(CUDA, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return [tuple(int(x) for x in line.split()) for line in out.splitlines()]


def test_eigensolver_clusters(tmp_path):
    """Never a larger cluster than the device places, an SM for each CTA of more than one per matrix,
    and on 152 SMs the bounds that were measured."""
    rows = _run(tmp_path, """
    for (int sms : {1, 7, 16, 60, 148, 152})
        for (int most : {8, 16})
            for (int n = 1; n <= 200; n++) std::printf("%d %d %d %d\\n", sms, most, n, jacobi_cluster(n, sms, most));
""")
    assert len(rows) == 6 * 2 * 200
    for sms, most, n, c in rows:
        assert c in (1, 2, 4, 8, 16) and c <= most
        assert c == 1 or n * c <= sms
    at = {(most, n): c for sms, most, n, c in rows if sms == 152}
    for n, c in ((1, 16), (8, 16), (9, 8), (18, 8), (19, 4), (38, 4), (39, 2), (76, 2), (77, 1)):
        assert at[16, n] == c and at[8, n] == min(c, 8)

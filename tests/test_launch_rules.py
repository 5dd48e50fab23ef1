"""Rules of the kernels and their launches that need no GPU, compiled from the library's own headers and
run on the host."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _run(tmp_path, body, headers=("pcsf_internal.h",), decl=""):
    """Output rows of a main() with this body: g++ for the host header, nvcc where device headers are in it."""
    cuh = any(h.endswith(".cuh") for h in headers)
    cc = (shutil.which("nvcc") or os.path.join(CUDA, "bin", "nvcc")) if cuh else shutil.which("g++")
    if cc is None or not os.path.exists(cc) or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no compiler or CUDA headers")
    src = tmp_path / ("rule.cu" if cuh else "rule.cpp")
    src.write_text("#include <cstdio>\n" + "".join('#include "%s"\n' % h for h in headers) +
                   "using namespace pcsf;\n%s\nint main()\n{\n%s\n}\n" % (decl, body))
    exe = tmp_path / "rule"
    flags = ["-gencode", "arch=compute_103a,code=sm_103a"] if cuh else []
    subprocess.run([cc, "-std=c++17"] + flags + ["-I", os.path.join(ROOT, "phylocsf_gb300", "csrc"), "-I",
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


def test_wait_for_the_last_contraction(tmp_path):
    """The parity that a leaving kernel waits for, against an mbarrier restated on the host (a wait for a
    parity returns at once unless the phase of that parity is the one in progress): it blocks exactly
    while the last contraction's commit is outstanding."""
    rows = _run(tmp_path, """
    for (int done = 0; done < 6; done++)               // contractions seen to complete
        for (int late = 0; late < 2; late++) {         // one more issued, its wait ran out
            ContractionPhase ph;
            uint32_t phase = 0;                        // the mbarrier's phase in progress
            for (int k = 0; k < done; k++) {
                phase++;                               // the commit arrives
                if ((phase & 1) == (ph.wait() & 1)) return 1;      // the wait would not return
                ph.next();
            }
            if (late) ph.next();
            std::printf("%d %d %d %d\\n", done, late, (phase & 1) == ph.last(), ((phase + 1) & 1) == ph.last());
        }
""", headers=("pcsf_internal.h", "prune_common.cuh", "tc_common.cuh"))
    assert len(rows) == 12
    for done, late, blocks, blocks_after in rows:
        assert blocks == late                          # waits while the commit is outstanding
        if late:
            assert not blocks_after                    # and no longer once it has arrived


def test_small_tiles(tmp_path):
    """FP32: up to four small tiles an SM.  FP64, in waves of long tiles (four small ones): while the last
    wave is at most three quarters full, in the third wave always, and up to four waves."""
    rows = _run(tmp_path, """
    for (int sms : {1, 7, 148, 152})
        for (int n = 0; n <= 17 * sms; n++) std::printf("%d %d %d %d\\n", sms, n, small_tiles(false, n, sms), small_tiles(true, n, sms));
""")
    assert len(rows) == 17 * (1 + 7 + 148 + 152) + 4
    for sms, n, fp32, fp64 in rows:
        assert fp32 == (n <= 4 * sms)
        quarters = -(-n // sms)               # of waves, the last one's begun
        assert fp64 == (quarters <= 16 and quarters not in (4, 8, 16))

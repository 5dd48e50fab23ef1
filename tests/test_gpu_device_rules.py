"""Arithmetic of the kernels that has a rule of its own, run on the device from the library's own headers
and compared there, value for value, with the plain expression that it stands for."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _run(tmp_path, headers, decl, body):
    """Whole numbers, by line, that a main() with this body prints."""
    nvcc = shutil.which("nvcc") or os.path.join(CUDA, "bin", "nvcc")
    src, exe = tmp_path / "rule.cu", tmp_path / "rule"
    src.write_text("#include <cmath>\n#include <cstdio>\n#include <vector>\n" + "".join('#include "%s"\n' % h for h in headers) +
                   "using namespace pcsf;\n%s\nint main()\n{\n%s\n}\n" % (decl, body))
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                    os.path.join(ROOT, "phylocsf_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    return [[int(x) for x in line.split()] for line in out.splitlines()]


# Spans of the operands' exponents: what a search meets, and up to where a quotient overflows or vanishes.
# No tolerance: each corrected operation is off by ~2^-88 before its rounding, so that one of ~2^35 rounds
# otherwise than the correctly rounded one, and 2^22 rotations have 2^24 operations.
@pytest.mark.parametrize("span", [3, 60, 290, 460, 790, 1000])
def test_rotation(tmp_path, span):
    rows = _run(tmp_path, ["jacobi_rotation.cuh"], """
constexpr int N = 1 << 22;
__device__ unsigned long long mix(unsigned long long z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
// +-m 2^e, m in [1, 2), |e| <= span; now and then a power of two
__device__ double draw(unsigned long long i, int span)
{
    const unsigned long long x = mix(i * 0x9E3779B97F4A7C15ull + span), y = mix(x);
    const double m = 1.0 + ((y & 15) ? (double)(x >> 12) * 0x1p-52 : 0.0);
    return ldexp((y >> 8) & 1 ? -m : m, (int)((y >> 16) % (2 * span + 1)) - span);
}
__global__ void check(int span, int *counts, double *first)
{
    const unsigned long long i = blockIdx.x * 256ull + threadIdx.x;
    double app = draw(3 * i, span), aqq = draw(3 * i + 1, span), apq = draw(3 * i + 2, span);
    if (i % 64 == 1) aqq = app;                     // a rotation by 45 degrees
    if (i % 64 == 2) app = 0.0;
    double c, s;
    jac_rotation(app, aqq, apq, c, s);
    const double theta = __ddiv_rn(aqq - app, 2.0 * apq);
    const double t = fabs(theta) > 1e150 ? 0.5 / theta
                     : __ddiv_rn(theta >= 0.0 ? 1.0 : -1.0, fabs(theta) + __dsqrt_rn(__fma_rn(theta, theta, 1.0)));
    const double rc = __ddiv_rn(1.0, __dsqrt_rn(__fma_rn(t, t, 1.0))), rs = t * rc;
    if (!isfinite(theta)) atomicAdd(counts + 1, 1);
    if (fabs(theta) < 0x1p300) atomicAdd(counts + 2, 1);
    if (!(c == rc && s == rs) && atomicAdd(counts, 1) == 0) {
        first[0] = app; first[1] = aqq; first[2] = apq; first[3] = c; first[4] = s; first[5] = rc; first[6] = rs;
    }
}
""", """
    int *counts;
    double *first;
    if (cudaMallocManaged(&counts, 3 * sizeof(int)) != cudaSuccess) return 1;
    if (cudaMallocManaged(&first, 7 * sizeof(double)) != cudaSuccess) return 1;
    for (int k = 0; k < 3; k++) counts[k] = 0;
    check<<<N / 256, 256>>>(SPAN, counts, first);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    if (counts[0]) for (int k = 0; k < 7; k++) std::fprintf(stderr, "%a\\n", first[k]);
    std::printf("%d %d %d\\n", counts[0], counts[1], counts[2]);
""".replace("SPAN", str(span)))
    wrong, infinite, common = rows[0]
    assert wrong == 0
    assert common > 0 and (infinite > 0) == (span >= 790)


def test_grid_point(tmp_path):
    """The grid point nearest to t, against the same rule with t's place found in FP64, at and around every
    grid point and midpoint, below the second point, beyond the last one and past the range of FP32."""
    rows = _run(tmp_path, ["pcsf_internal.h", "prune_common.cuh"], """
__global__ void check(DevModels m, const double *t, int n, int *counts)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n || t[i] < m.grid_t[0]) return;
    const double x = floor(log(t[i] / m.grid_t[0]) / m.grid_lr);
    int g = x < 0.0 ? 0 : x > m.grid_n - 1 ? m.grid_n - 1 : (int)x;
    if (g + 1 < m.grid_n && (m.grid_t[g + 1] - t[i]) < (t[i] - m.grid_t[g])) g++;
    atomicAdd(counts, 1);
    if (grid_point(m, t[i]) != g) atomicAdd(counts + 1, 1);
}
""", """
    const int G = 6500;
    const double lr = std::log(1.002), rel[] = {0, 1e-16, 1e-13, 1e-10, 1e-8, 1e-7, 1e-6, 1e-5, 3e-4};
    std::vector<double> grid(G), ts = {1e-3, 1.0, 1e30, 1e38, 1e39, 1e200, 1e308};
    for (int g = 0; g < G; g++) grid[g] = 1e-5 * std::exp(lr * g);
    for (int g = 0; g < G; g++)
        for (double r : rel)
            for (double sign : {1.0, -1.0}) {
                ts.push_back(grid[g] * (1.0 + sign * r));
                if (g) ts.push_back(0.5 * (grid[g] + grid[g - 1]) * (1.0 + sign * r));
            }
    const int n = (int)ts.size();
    DevModels m{};
    double *dg, *dt;
    int *counts;
    if (cudaMallocManaged(&dg, G * sizeof(double)) != cudaSuccess) return 1;
    if (cudaMallocManaged(&dt, n * sizeof(double)) != cudaSuccess) return 1;
    if (cudaMallocManaged(&counts, 2 * sizeof(int)) != cudaSuccess) return 1;
    for (int k = 0; k < G; k++) dg[k] = grid[k];
    for (int k = 0; k < n; k++) dt[k] = ts[k];
    counts[0] = counts[1] = 0;
    m.grid_t = dg;
    m.grid_n = G;
    m.grid_lr = lr;
    check<<<(n + 255) / 256, 256>>>(m, dt, n, counts);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    std::printf("%d %d\\n", counts[0], counts[1]);
""")
    compared, wrong = rows[0]
    assert compared > 200_000 and wrong == 0

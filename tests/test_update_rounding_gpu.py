"""The update of one point and of two points per instruction round alike whatever the compiler
contracts: st_update.cuh built with and without contraction, on values of many magnitudes, bit
for bit."""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "st_update.cuh"
#include <cstdio>
#include <vector>
using namespace stg;
__global__ void both(const float* in, float* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* v = in + 13 * i;  // u D pv xm xp ym yp zm zp c ax ay az
    const float upd = v[1] * v[2];
    out[3 * i] = update_fast(v[0], upd, v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], v[11], v[12]);
    F2 r = update2(pack(v[0], v[0]), pack(-v[1], -v[1]), pack(v[2], v[2]), add2(pack(v[4], v[4]), pack(v[3], v[3])),
                   add2(pack(v[6], v[6]), pack(v[5], v[5])), add2(pack(v[8], v[8]), pack(v[7], v[7])), pack(v[9], v[9]),
                   v[10], v[11], v[12]);
    unpack(r, out[3 * i + 1], out[3 * i + 2]);
}
int main(int argc, char** argv) {
    const int n = atoi(argv[1]);
    std::vector<float> in(13 * n), out(3 * n);
    FILE* f = fopen(argv[2], "rb");
    if (!f || fread(in.data(), 4, in.size(), f) != in.size()) return 1;
    fclose(f);
    float *a, *b;
    if (cudaMalloc(&a, in.size() * 4) || cudaMalloc(&b, out.size() * 4)) return 2;
    cudaMemcpy(a, in.data(), in.size() * 4, cudaMemcpyHostToDevice);
    both<<<(n + 255) / 256, 256>>>(a, b, n);
    if (cudaMemcpy(out.data(), b, out.size() * 4, cudaMemcpyDeviceToHost)) return 3;
    f = fopen(argv[3], "wb");
    return fwrite(out.data(), 4, out.size(), f) == out.size() && !fclose(f) ? 0 : 4;
}
"""


@pytest.mark.parametrize("fmad", ["true", "false"])
def test_scalar_and_packed_forms_agree(tmp_path, fmad):
    import importlib.util
    pkg = os.path.join(ROOT, "03-seismic-tomography-compute_gb300")
    spec = importlib.util.spec_from_file_location("st_build", os.path.join(pkg, "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    src, exe, fin, fout = (str(tmp_path / n) for n in ("u.cu", "u", "in", "out"))
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([b.nvcc(), *b.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", f"-fmad={fmad}", "-I", b.INCLUDE,
                    "-I", b.CSRC, src, "-o", exe], check=True, capture_output=True)
    n = 100_000
    rng = np.random.default_rng(5)
    v = (rng.standard_normal((n, 13)) * 10.0 ** rng.integers(-6, 3, (n, 1))).astype(np.float32)
    v[:, 1] = rng.random(n)
    v[:, 9:] = rng.random((n, 4)) + 0.01
    v.tofile(fin)
    subprocess.run([exe, str(n), fin, fout], check=True)
    out = np.fromfile(fout, np.float32).reshape(n, 3)
    assert np.array_equal(out[:, 0], out[:, 1]) and np.array_equal(out[:, 0], out[:, 2])
    assert np.isfinite(out).all() and np.abs(out).max() > 0

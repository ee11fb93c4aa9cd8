"""The reciprocal of the symmetry-adapted Euler kernel (recip in
csrc/dglm_stage_sym.cuh), compiled on its own, against IEEE division on the
host: within one ulp for normal x below 2^1022 of either sign.  (Derived: the
approximation is good to 2^-23, two Newton steps square that twice, and the
last fma rounds once, so the error is half an ulp and a few 2^-90.)  NaN for 0,
subnormal numbers, infinities and NaN."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from exadglm_b200 import build as _build

SOURCE = r"""
#include "dglm_sym.cuh"
__global__ void run(const double *x, double *y, long n) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) y[i] = dglm::recip(x[i]);
}
extern "C" int recip(const double *x, double *y, long n) {
  run<<<(unsigned)((n + 255) / 256), 256>>>(x, y, n);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.mark.gpu
def test_reciprocal(tmp_path):
    torch = pytest.importorskip("torch")
    src, lib = tmp_path / "recip.cu", tmp_path / "librecip.so"
    src.write_text(SOURCE)
    subprocess.run([_build.nvcc(), *_build.ARCH, *_build.NVCC_FLAGS, "-shared", "-cudart",
                    "static", "-o", str(lib), str(src)], check=True)
    f = C.CDLL(str(lib)).recip
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_long]
    rng = np.random.default_rng(0)
    mant = np.concatenate([1 + rng.random(2000), [1.0, 2 - 2.0 ** -52, 1.5, 1 + 2.0 ** -52]])
    x = (mant[None, :] * 2.0 ** np.arange(-1022, 1022)[:, None].astype(float)).ravel()
    x = np.concatenate([x, -x])
    odd = np.array([0.0, -0.0, 5e-324, 2.0 ** -1023, np.inf, -np.inf, np.nan])

    def run(a):
        d = torch.from_numpy(np.ascontiguousarray(a)).cuda()
        out = torch.empty_like(d)
        assert f(d.data_ptr(), out.data_ptr(), d.numel()) == 0
        return out.cpu().numpy()

    got, want = run(x), 1.0 / x
    ulps = np.abs(got.view(np.int64) - want.view(np.int64))
    print("worst", ulps.max(), "ulp;", (ulps > 0).mean(), "of the results differ")
    assert ulps.max() <= 1
    assert np.isnan(run(odd)).all()

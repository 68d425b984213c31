"""exact_div.cuh's reciprocals and quotients against CUDA's own IEEE division,
bit for bit: over the documented ranges and at their ends, for all-ones and
other extreme significands, quotients next to rounding boundaries, signed
zeros and random operands."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "exact_div.cuh"
// which: 0 recip_rn(b), 1 quot_pos(a, b), 2 quot(a, b); bad: mismatches, first: lowest mismatching index
__global__ void check(const double* a, const double* b, long long n, int which, unsigned long long* bad,
                      unsigned long long* first) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double x = a[i], y = b[i];
        const double got = which == 0 ? bsn::f64::recip_rn(y)
                         : which == 1 ? bsn::f64::quot_pos(x, y, bsn::f64::recip_rn(y))
                                      : bsn::f64::quot(x, y, bsn::f64::recip_rn(fabs(y)));
        const double want = which == 0 ? 1.0 / y : x / y;
        if (__double_as_longlong(got) != __double_as_longlong(want)) {
            atomicAdd(bad, 1ull);
            atomicMin(first, (unsigned long long)i);
        }
    }
}
extern "C" int run(const double* a, const double* b, long long n, int which, unsigned long long* out) {
    check<<<592, 256>>>(a, b, n, which, out, out + 1);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def mismatches(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact_div")
    (d / "check.cu").write_text(SOURCE)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "-prec-div=true", "-Xcompiler", "-fPIC", "-shared",
                    "-I" + os.path.join(ROOT, "binary-supernova_b200", "csrc"), "-o", str(d / "check.so"),
                    str(d / "check.cu"), "-lcudart"], check=True)
    L = C.CDLL(str(d / "check.so"))

    def run(a, b, which):
        a, b = np.broadcast_arrays(np.asarray(a, np.float64), np.asarray(b, np.float64))
        A, B = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (a, b))
        out = torch.tensor([0, 2 ** 62], dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        assert L.run(C.c_void_p(A.data_ptr()), C.c_void_p(B.data_ptr()), C.c_longlong(A.numel()), which,
                     C.c_void_p(out.data_ptr())) == 0
        bad, first = out.tolist()
        return 0 if not bad else (bad, a[first].hex(), b[first].hex())
    return run


def _significands(rng, n):
    """In [1, 2): the extremes, all but a few leading or trailing bits set or clear, and random ones."""
    m = [0, 1, 2, 3, 2 ** 52 - 1, 2 ** 52 - 2, 2 ** 52 - 3, 2 ** 51, 2 ** 51 - 1, 2 ** 51 + 1]
    m += [2 ** 52 - 2 ** k for k in range(52)] + [2 ** k - 1 for k in range(52)]
    m = np.concatenate([np.array(m, dtype=np.int64), rng.integers(0, 2 ** 52, n - len(m))])
    return (m + (1023 << 52)).view(np.float64)


def test_reciprocals(mismatches):
    rng = np.random.default_rng(1)
    s = _significands(rng, 4096)
    for e in (-340, -339, -100, -1, 0, 1, 116, 300, 738, 739):
        assert not mismatches(1.0, np.ldexp(s, e), 0)
    s = _significands(rng, 4_000_000)
    assert not mismatches(1.0, np.ldexp(s, rng.integers(-340, 740, s.size)), 0)


@pytest.mark.parametrize("which", [1, 2])
def test_quotients(mismatches, which):
    rng = np.random.default_rng(2)
    sign = (lambda n: rng.choice([-1.0, 1.0], n)) if which == 2 else (lambda n: np.ones(n))
    n = 4_000_000
    # random operands, denominators over their range, quotients that stay normal
    b = np.ldexp(_significands(rng, n), rng.integers(-340, 300, n))
    eq = rng.integers(-560, 600, n)
    a = np.ldexp(rng.permutation(_significands(rng, n)), np.clip(np.frexp(b)[1] + eq, -900, 1000))
    assert not mismatches(sign(n) * a, sign(n) * b, which)
    # numerators next to b times a rounding boundary (half an ulp above a double)
    s, t = _significands(rng, n), rng.permutation(_significands(rng, n))
    near = s * t + s * 2.0 ** -53
    for k in (-1, 0, 1):
        x = near + k * np.spacing(near)
        e = rng.integers(-300, 300, n)
        assert not mismatches(sign(n) * np.ldexp(x, e), sign(n) * s, which)
    # the ends of the numerators' range, all pairs of extreme significands
    s = _significands(rng, 200)
    for ea, eb in ((-900, -340), (-900, 100), (-600, 299), (115, -340), (400, -340), (0, 0), (399, 299)):
        x, y = np.ldexp(np.repeat(s, 200), ea), np.ldexp(np.tile(s, 200), eb)
        assert not mismatches(sign(x.size) * x, sign(x.size) * y, which)
    # zeros
    z = np.concatenate([np.zeros(200), -np.zeros(200)]) if which == 2 else np.zeros(400)
    assert not mismatches(z, np.tile(s, 2), which)
    if which == 2:
        assert not mismatches(z, -np.tile(s, 2), which)

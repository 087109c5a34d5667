"""The quotients that the 3-D kernels form without a division are the IEEE-rounded ones: the passes'
harmonic buoyancy means (a Newton step on the hardware reciprocal, then Markstein's correction of the
quotient) over the admissible densities, and the volume renderer's shared divisors over its ranges,
infinite quotients among them.  Bit for bit against the device's IEEE division.

For the means the reciprocal after the Newton step is the rounded one, whatever the hardware's is within
its 1 ulp, but for 32 of the 2^23 mantissas of the sum a + b (HARD, found by trying all of them);
for these a sweep of all numerators leaves a doubt at one numerator of two mantissas."""
import ctypes
import os
import shutil
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
PAIRS = 1 << 26
HARD = [0x069913, 0x07cc45, 0x0efa43, 0x109909, 0x186799, 0x1beaaf, 0x20ddd1, 0x224cf7, 0x26449f, 0x2aaaac, 0x2b8be1,
        0x2d1367, 0x384a93, 0x423dc3, 0x50ac19, 0x50dd0d, 0x525d25, 0x543d43, 0x5c23dd, 0x5e86a9, 0x605475, 0x61368b,
        0x625473, 0x6c7ec7, 0x6e4bc5, 0x700ff1, 0x702a3b, 0x70ff0f, 0x7c3237, 0x7e01ff, 0x7ffffd, 0x7fffff]


@pytest.fixture(scope="module")
def check(tmp_path_factory, cuda_device):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no CUDA compiler")
    out = str(tmp_path_factory.mktemp("division") / "division_check.so")
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-Xcompiler", "-fPIC", "-shared",
                    "-o", out, os.path.join(HERE, "division_check.cu")], check=True)
    fn = ctypes.CDLL(out).division_check
    fn.restype, fn.argtypes = ctypes.c_longlong, [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong]

    def run(means, a, b):
        assert a.dtype == b.dtype == torch.float32 and a.is_contiguous() and b.is_contiguous()
        assert a.is_cuda and b.is_cuda and a.numel() == b.numel() and a.numel() % 2 == 0
        torch.cuda.synchronize()
        return fn(int(means), a.data_ptr(), b.data_ptr(), a.numel())

    return run


def spread(low, high, seed, signed=False):
    """Values spread evenly over the logarithm of [low, high]."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(PAIRS, dtype=torch.float64, device="cuda", generator=g)
    v = torch.exp2(u * (torch.log2(torch.tensor(high / low, dtype=torch.float64)).item())) * low
    if signed:
        v = torch.where(torch.rand(PAIRS, device="cuda", generator=g) < 0.5, -v, v)
    return v.float()


def from_bits(bits):
    return bits.to(torch.int32).view(torch.float32)


@pytest.mark.parametrize("low,high", [(1000.0, 5000.0), (1.0, 50000.0), (1e-17, 50000.0)])
def test_buoyancy_means(low, high, check):
    a, b = 1.0 / spread(low, high, 1), 1.0 / spread(low, high, 2)
    assert check(True, a, b) == 0


def test_buoyancy_means_of_every_mantissa(check):
    bits = torch.arange(1 << 23, device="cuda") | 0x3A000000       # 1/2048 .. 1/1024
    a = from_bits(bits)
    assert check(True, a, a) == 0
    assert check(True, a, a.flip(0).contiguous()) == 0


def test_buoyancy_means_of_hard_sums(check):
    g = torch.Generator(device="cuda").manual_seed(3)
    for m in HARD:
        total = from_bits(torch.full((1 << 21,), 0x3A800000 | m, device="cuda"))
        a = torch.rand(1 << 21, device="cuda", generator=g) * total
        b = total - a
        keep = (a > 0) & (b > 0) & (a + b == total)
        a, b = a[keep], b[keep]
        n = a.numel() // 2 * 2
        assert n > 1 << 18
        assert check(True, a[:n].contiguous(), b[:n].contiguous()) == 0


# Numerators and divisors: ray positions over extents, wave values over the display scale, magnitudes over
# the threshold's span, materials over their range, colours over densities.
@pytest.mark.parametrize("x,d", [((1e-6, 4.0), (1e-3, 1.0)), ((1e-25, 1e10), (1e-20, 1e10)), ((1e-12, 1e6), (1e-6, 1.0)),
                                 ((1e-3, 5e4), (1e-6, 5e4)), ((1e-20, 1e3), (1e-10, 1e3)), ((0.999, 1.001), (0.999, 1.001))])
def test_renderer_quotients(x, d, check):
    assert check(False, spread(*x, 4, signed=True), spread(*d, 5)) == 0


def test_renderer_quotients_that_overflow(check):
    x, d = spread(1e28, 3.4e38, 6, signed=True), spread(1e-20, 1e-11, 7)
    assert check(False, x, d) == 0
    x[::3] = float("inf")
    x[1::3] = -float("inf")
    assert check(False, x, d) == 0
    x[:] = 0.0
    assert check(False, x, d) == 0

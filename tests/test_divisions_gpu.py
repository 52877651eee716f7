"""The divisions without a branch behind sigmoid and SiLU (``gb::over``, ``gb::divide``) give the division's own bits: every denominator
from 1 up (all but five beyond 2^126), SiLU's quotient for every 32-bit number, quotients of other numbers down to the line that the kernels'
header draws."""
import pytest
import torch

pytestmark = pytest.mark.gpu
STEP = 1 << 24


@pytest.fixture(scope="module")
def divide():
    from garuda_b200.kernels.ops import CudaOps
    return CudaOps("cuda:0").selftest_divisions


def floats(bits):
    return bits.to(torch.int32).view(torch.float32)


def differ(a, b):
    """How many differ in a bit (of what is not a number, any is alike)."""
    return int(((a.view(torch.int32) != b.view(torch.int32)) & ~(a.isnan() & b.isnan())).sum())


def test_every_reciprocal(divide):
    first, subnormal, last, off = 0x3f800000, 0x7e800000, 0x7f800000, 0             # 1, 2^126, infinity
    for at in range(first, last + 1, STEP):
        d = floats(torch.arange(at, min(at + STEP, last + 2), device="cuda"))        # (one beyond infinity is not a number)
        got, want = divide(d, d)[1], torch.ones_like(d) / d
        if at < subnormal:
            assert differ(got, want) == 0
        else:                                               # Newton's step leaves those next to the middle between two numbers a last place off
            off += differ(got, want)
            near = ~want.isnan()
            assert ((got[near].view(torch.int32) - want[near].view(torch.int32)).abs() <= 1).all() and got[~near].isnan().all()
    assert off <= 5


def test_every_silu(divide):
    off = 0
    for at in range(0, 1 << 32, STEP):
        z = floats(torch.arange(at, at + STEP, device="cuda"))
        d = 1.0 + torch.exp(-z)
        off += differ(divide(z, d)[0], z / d)
    assert off == 0


@pytest.mark.parametrize("smallest", [2.0 ** -100, 1.0])
def test_other_quotients(divide, smallest):
    g = torch.Generator(device="cuda").manual_seed(3)
    for _ in range(8):
        sign = torch.randint(0, 2, (STEP,), generator=g, device="cuda") * 2.0 - 1.0
        z = sign * smallest * torch.exp2(torch.rand(STEP, generator=g, device="cuda") * 30)
        d = torch.exp2(torch.rand(STEP, generator=g, device="cuda") * 24)
        assert differ(divide(z, d)[0], z / d) == 0

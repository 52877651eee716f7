"""The 32-bit kernels in tiles: the matrix product at the edges of its tiles and of its parts of K, whose
numbers must not depend on how many rows it has; the prompt attention, which must give the plain kernel's
bits whatever lies in the cache behind a query's own position."""
import pytest
import torch

from tests.test_kernels_gpu import _attention_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plain():
    from garuda_b200.kernels import CudaOps
    return CudaOps("cuda:0", tensor_cores=False)


# (N, K): K of one block at most and K % 4 != 0 (the older kernel); one tile, K in one part; a tail of both; eight parts; parts of unequal length; two
# parts; many tiles; tiles of 16, 32 and 64 rows for the most rows
@pytest.mark.parametrize("N,K", [(128, 16), (130, 20), (96, 32), (96, 70), (128, 36), (130, 44), (256, 1024), (2000, 1284), (11264, 256), (24000, 64),
                                 (16, 192), (6000, 40), (8192, 100)])
def test_product_over_row_counts(plain, N, K):
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a, w = torch.randn(200, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda") * 0.1
    base = torch.randn(200, N, generator=g, device="cuda")
    ref = a.double() @ w.double().t()
    # K products of 24-bit numbers, added in parts of at most K: the rounding of a sum grows as the root of its length
    tol = 2e-6 * max(1.0, (K / 256) ** 0.5)
    whole = None
    for M in (200, 65, 64, 33, 32, 17, 16, 9, 8, 1):
        out, acc = torch.full((M, N), float("nan"), device="cuda"), base[:M].clone()
        plain.linear(a[:M], w, out)
        plain.linear(a[:M], w, acc, accumulate=True, alpha=0.5)
        scale = ref.abs().max()
        assert (out.double() - ref[:M]).abs().max() <= tol * scale
        assert (acc.double() - base[:M].double() - 0.5 * ref[:M]).abs().max() <= tol * scale
        whole = out if whole is None else whole
        assert torch.equal(out, whole[:M]), f"{M} rows"


def test_product_of_an_unaligned_operand(plain):
    """Rows that do not start on 16 bytes take the kernel that reads number by number."""
    a, w = torch.randn(1 + 9 * 64, device="cuda")[1:].view(9, 64), torch.randn(100, 64, device="cuda")
    out = torch.zeros(9, 100, device="cuda")
    plain.linear(a, w, out)
    assert (out - (a.double() @ w.double().t())).abs().max() <= 1e-5 * out.abs().max()


@pytest.mark.parametrize("Hq,Hkv,hd,page,reqs", [(32, 4, 64, 32, [(125, 125), (375, 375)]), (8, 8, 128, 16, [(97, 33), (32, 32), (64, 1)]),
                                                 (6, 2, 64, 8, [(300, 45), (31, 31), (33, 33)]), (4, 1, 128, 32, [(1000, 129)]), (5, 1, 64, 4, [(70, 64)])])
def test_prompt_attention_gives_the_plain_kernels_bits(plain, Hq, Hkv, hd, page, reqs):
    q, k, v, bt, cu, kvl, treq, ref = (t.cuda() for t in _attention_case(Hq, Hkv, hd, page, reqs, 0, torch.float32))
    # what lies behind a request's last position may be anything
    for r, (kv, _) in enumerate(reqs):
        if kv % page:
            for pool in (k, v):
                pool[bt[r, kv // page].long(), :, kv % page:] = float("nan")
    bt[0, 1] = -1                                    # a page that was given back
    out, other = torch.zeros_like(ref), torch.full_like(ref, float("nan"))
    before = plain.launches
    plain.paged_attention(q, k, v, bt, cu, kvl, treq, out, hd ** -0.5, 0, page, len(reqs), max(n for _, n in reqs), max(n for n, _ in reqs))
    assert plain.launches == before + 1
    L = plain.core
    assert L.gb_attention_simple(q.data_ptr(), k.data_ptr(), v.data_ptr(), 0, bt.data_ptr(), bt.shape[1], cu.data_ptr(), kvl.data_ptr(), treq.data_ptr(),
                                 other.data_ptr(), q.shape[0], Hq, Hkv, hd, hd, hd, hd ** -0.5, 0, page, 0.0, 0, 0, None, None, None, 0,
                                 plain._stream()) == 0
    torch.cuda.synchronize()
    assert torch.isfinite(other).all() and torch.equal(out, other)


def test_prompt_attention_of_a_later_token_that_is_not_a_number(plain):
    Hq, Hkv, hd, page, n = 8, 2, 64, 16, 90
    q, k, v, bt, cu, kvl, treq, _ = (t.cuda() for t in _attention_case(Hq, Hkv, hd, page, [(n, n)], 0, torch.float32))
    outs = []
    for spoil in (False, True):
        if spoil:
            k[bt[0, 50 // page].long(), :, 50 % page] = float("nan")
            v[bt[0, 70 // page].long(), :, 70 % page] = float("inf")
        out = torch.zeros(n, Hq * hd, device="cuda")
        plain.paged_attention(q, k, v, bt, cu, kvl, treq, out, hd ** -0.5, 0, page, 1, n, n)
        outs.append(out)
    assert torch.equal(outs[0][:50], outs[1][:50])

"""Rows that leave 16 bytes at a time, and rows that cannot: a fused projection's split into queries and pages, the per-head products."""
import pytest
import torch

from tests.gpu_helpers import close, rnd

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from garuda_b200.kernels.ops import CudaOps
    return CudaOps("cuda:0")


# widths in fours, one width that is not, a row beyond one pass of the block, operands that do not start on 16 bytes
@pytest.mark.parametrize("Hq,Hkv,hd,vd,shift", [(3, 2, 24, 40, 0), (1, 1, 4, 4, 0), (5, 1, 6, 10, 0), (3, 2, 24, 42, 0), (40, 8, 64, 64, 0), (3, 2, 24, 40, 1)])
@pytest.mark.parametrize("dt,biased", [(torch.bfloat16, True), (torch.float32, False)])
def test_split_into_pages(ops, Hq, Hkv, hd, vd, shift, dt, biased):
    from tests.plain.cpu_ops import CpuOps
    T, page, cols = 9, 8, Hq * hd + Hkv * (hd + vd)
    qkv, bias = rnd(T, cols), rnd(cols, seed=1) if biased else None
    pos = torch.tensor([6, 7, 8, 0, 31, 32, 3, 0, 5], dtype=torch.int32)
    req = torch.tensor([0, 0, 0, 1, 2, 2, 3, 3, 1], dtype=torch.int32)
    table = torch.tensor([[4, 1, -1, -1, -1], [0, -1, -1, -1, -1], [-1, -1, -1, 2, 5], [-1, -1, -1, -1, -1]], dtype=torch.int32)
    place = lambda *shape: torch.zeros(shape, dtype=dt)
    outs = [place(T, Hq, hd), place(6, Hkv, page, hd), place(6, Hkv, page, vd)]
    got = [torch.zeros(o.numel() + shift, dtype=dt, device="cuda")[shift:].view(o.shape) for o in outs]
    ops.qkv_bias_append(qkv.cuda(), None if bias is None else bias.cuda(), *got, pos.cuda(), req.cuda(), table.cuda(), Hq, Hkv, hd, vd, page)
    CpuOps().qkv_bias_append(qkv, bias, *outs, pos, req, table, Hq, Hkv, hd, vd, page)
    for a, b in zip(got, outs):
        assert torch.equal(a.cpu(), b)


# the edges of tiles of rows and columns; columns that are no multiple of eight; a view whose rows start on 4 bytes
@pytest.mark.parametrize("T", [1, 17, 64, 130])
@pytest.mark.parametrize("n,k,lead", [(256, 32, 0), (264, 64, 0), (8, 8, 0), (20, 32, 0), (64, 40, 2)])
def test_per_head_products(ops, T, n, k, lead):
    H, bf = 3, torch.bfloat16
    a, w = rnd(T, H, k, dtype=bf), rnd(H * n, k, dtype=bf, scale=k ** -0.5, seed=1)
    room = torch.full((T, H, n + 8), float("nan"), dtype=bf, device="cuda")
    ops.head_linear(a.cuda(), w.cuda(), room[:, :, lead:lead + n], n, k, False)
    want = torch.einsum("thk,hnk->thn", a.double(), w.view(H, n, k).double())
    close(room[:, :, lead:lead + n], want, bf, "per-head products", tol=2 ** -8)      # half of bfloat16's last place, of the largest
    assert room[:, :, :lead].isnan().all() and room[:, :, lead + n:].isnan().all(), "a store beyond the row"

"""Attention over cached latent rows for prompt portions on the tcgen05 kernel, against 64-bit attention over
the same rows: every block count of a row (with and without a rotated part that fills its block), one tile of
64 keys and its edges, portions behind cached positions, single tokens beside them, pages of every size, sinks, whatever
lies behind a request's last position."""
import pytest
import torch

from tests.gpu_helpers import close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from garuda_b200.kernels.ops import CudaOps
    return CudaOps("cuda:0")


# (rank, rot, heads, page size, (cached length after the step, tokens of the step) of every request, sinks)
@pytest.mark.parametrize("rank,rot,H,page,reqs,sinks", [
    (256, 32, 32, 32, [(300, 300)], False), (256, 64, 16, 16, [(64, 64), (65, 65), (700, 350), (129, 1)], True),
    (64, 32, 32, 8, [(333, 333), (63, 63)], False), (128, 0, 24, 64, [(1000, 340), (128, 128)], True), (192, 16, 40, 32, [(2111, 200)], False),
    # decoded tokens, on either side of the line between the two kernels
    (64, 32, 16, 8, [(40 + i % 100, 1) for i in range(130)], True), (64, 32, 16, 8, [(40 + i % 100, 1) for i in range(200)], True),
    (256, 32, 32, 32, [(400 - i % 90, 1) for i in range(170)], False), (256, 32, 32, 32, [(200 - i % 90, 1) for i in range(170)], True),
    (256, 32, 8, 16, [(1024 + i % 70, 1) for i in range(150)], False)])
def test_prompt_portions(ops, rank, rot, H, page, reqs, sinks):
    row, R = rank + rot, len(reqs)
    g = torch.Generator(device="cuda").manual_seed(rank + rot)
    T = sum(n for _, n in reqs)
    each = [(kv + page - 1) // page for kv, _ in reqs]
    pool = torch.full((sum(each) + 3, 1, page, row), float("nan"), dtype=torch.bfloat16, device="cuda")      # what nobody wrote
    order = torch.randperm(sum(each) + 3, generator=g, device="cuda").int()
    table = torch.full((R, max(each) + 1), -1, dtype=torch.int32, device="cuda")
    q = torch.randn(T, H, row, generator=g, device="cuda").bfloat16()
    sink = torch.randn(H, generator=g, device="cuda") + 2.0 if sinks else None
    scale, at, t0, ref = row ** -0.5, 0, 0, torch.empty(T, H, rank, dtype=torch.float64, device="cuda")
    for r, (kv, n) in enumerate(reqs):
        table[r, :each[r]] = order[at:at + each[r]]
        rows = torch.randn(kv, row, generator=g, device="cuda").bfloat16()
        j = torch.arange(kv, device="cuda")
        pool[table[r].long()[j // page], 0, j % page] = rows
        s = torch.einsum("thc,jc->htj", q[t0:t0 + n].double(), rows.double()) * scale
        s = s.masked_fill(j[None, None, :] > (kv - n + torch.arange(n, device="cuda"))[None, :, None], -float("inf"))
        e = torch.exp(s - s.amax(-1, keepdim=True))
        den = e.sum(-1, keepdim=True) + (torch.exp(sink.double()[:, None, None] - s.amax(-1, keepdim=True)) if sinks else 0.0)
        ref[t0:t0 + n] = torch.einsum("htj,jc->thc", e / den, rows[:, :rank].double())
        at, t0 = at + each[r], t0 + n
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu = i32([sum(n for _, n in reqs[:r]) for r in range(R + 1)])
    out = torch.full((T, H * rank), float("nan"), dtype=torch.bfloat16, device="cuda")
    lib = ops.tc._latent_lib(rank, rot)
    assert lib.gb_latent_attention_tc_takes(q.data_ptr(), pool.data_ptr(), out.data_ptr(), page, pool.shape[0], T * H) == 1
    assert ops.tc.latent_plan(R, H, max(n for _, n in reqs), max(kv for kv, _ in reqs)) == 1
    req = torch.repeat_interleave(torch.arange(R, dtype=torch.int32), torch.tensor([n for _, n in reqs])).cuda()
    more = {} if sink is None else dict(sink_values=sink)
    ops.paged_attention(q, pool, pool, table, cu, i32([kv for kv, _ in reqs]), req, out, scale, 0, page, R, max(n for _, n in reqs),
                        max(kv for kv, _ in reqs), value_dim=rank, **more)
    ops.tc.check_errors()
    close(out.view(T, H, rank), ref.cpu(), torch.bfloat16, "latent attention")


def test_the_largest_weight_is_not_rounded(ops):
    """Every value is one and two keys have a weight: the result is one, whatever the later key's score is above the earlier one's. Its
    weight, taken against any other score than the largest, would be rounded to bfloat16 and be off by up to a 256th."""
    rank, rot, H, page, n, late = 256, 32, 32, 32, 600, 70
    pool = torch.zeros(n // page + 1, 1, page, rank + rot, dtype=torch.bfloat16, device="cuda")
    flat = pool.view(-1, rank + rot)
    flat[:, :rank], flat[:, rank], flat[0, rank], flat[late, rank] = 1.0, -1000.0, 0.0, 1.0
    q = torch.zeros(n, H, rank + rot, dtype=torch.bfloat16, device="cuda")
    q[:, :, rank] = torch.linspace(0.1, 5.5, n * H, device="cuda").view(n, H).bfloat16()      # 0.14 to 7.9 powers of two
    table = torch.arange(n // page + 1, dtype=torch.int32, device="cuda")[None]
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    out = torch.full((n, H * rank), float("nan"), dtype=torch.bfloat16, device="cuda")
    assert ops.tc._latent_lib(rank, rot).gb_latent_attention_tc_takes(q.data_ptr(), pool.data_ptr(), out.data_ptr(), page, pool.shape[0], n * H) == 1
    ops.paged_attention(q, pool, pool, table, i32(0, n), i32(n), torch.zeros(n, dtype=torch.int32, device="cuda"), out, 1.0, 0, page, 1, n, n, value_dim=rank)
    ops.tc.check_errors()
    assert torch.equal(out, torch.ones_like(out))


@pytest.mark.parametrize("what", ["nan", "inf"])
def test_a_cached_row_that_is_not_finite(ops, what):
    """Every row that reads it is not a number; those in front of its tile of 128 query rows are as if it were not there."""
    rank, rot, H, page, n, bad = 64, 32, 32, 16, 300, 150
    g = torch.Generator(device="cuda").manual_seed(5)
    q, pool = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((n, H, rank + rot), (n // page + 1, 1, page, rank + rot)))
    q[..., 0] = q[..., 0].abs() + 0.5                     # a score of plus infinity, not minus
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    table, outs = torch.arange(n // page + 1, dtype=torch.int32, device="cuda")[None], []
    for value in (None, float(what)):
        if value is not None:
            pool[bad // page, 0, bad % page, 0] = value
        outs.append(torch.zeros(n, H * rank, dtype=torch.bfloat16, device="cuda"))
        ops.paged_attention(q, pool, pool, table, i32(0, n), i32(n), torch.zeros(n, dtype=torch.int32, device="cuda"), outs[-1], 0.1, 0, page, 1, n, n,
                            value_dim=rank)
    first = bad * H // 128 * 128 // H                     # the tile's first token
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0][:first], outs[1][:first])
    assert torch.isnan(outs[1][bad:].view(-1, H, rank)).all()


@pytest.mark.parametrize("rank,H,lens,kv,tcgen05", [
    (256, 32, [300], 300, True), (256, 8, [1] * 148, 70, True), (256, 8, [1] * 149, 1023, False), (256, 8, [1] * 149, 1024, True),
    (256, 32, [1] * 149, 255, False), (256, 32, [1] * 149, 256, True), (64, 64, [1] * 149, 4000, False), (64, 16, [60, 1, 1, 1], 4000, True),
    (64, 16, [200] + [1] * 200, 1200, False), (64, 32, [90] * 16, 90, False), (64, 32, [97] * 16, 97, True), (256, 64, [45] * 16, 45, True)])
def test_which_kernel(ops, rank, H, lens, kv, tcgen05):
    assert ops.tc.latent_on_tcgen05(rank, sum(lens), len(lens), H, max(lens), kv, 148) == tcgen05

"""Products of some hundreds of tokens in token blocks by 256 features with K split over a cluster's pairs, against plain 32-bit
products: one and two parts a block, one and several blocks, every split from one to four, features that fill no pair of CTAs, a K that is no
multiple of a step, and each epilogue: stored, stored through each activation, added, added with the next norm folded in, rotated into
pages, and rotated behind a folded norm."""
import pytest
import torch

from tests.gpu_helpers import close, rnd

pytestmark = pytest.mark.gpu

# tokens, features, K
SHAPES = [(257, 264, 2048), (333, 4096, 4104), (384, 1000, 2048), (511, 2048, 5632), (512, 18560, 4096), (513, 2048, 5632), (1030, 4096, 2048),
          (1221, 4096, 2048), (300, 288, 2040), (270, 2500, 4104), (2262, 700, 4096)]


@pytest.fixture(scope="module")
def ops():
    from garuda_b200.kernels.ops import CudaOps
    torch.backends.cuda.matmul.allow_tf32 = False
    return CudaOps("cuda:0", tensor_cores=True)


def operands(M, N, K, seed=0):
    a = rnd(M, K, scale=0.5, seed=seed).cuda().bfloat16()
    w = rnd(N, K, scale=K ** -0.5, seed=seed + 1).cuda().bfloat16()
    return a, w, a.float() @ w.float().T


def test_the_shapes_take_the_kernel(ops):
    splits = [ops.tc.lib.gb_gemm_tc_tall(*s) for s in SHAPES]
    assert set(splits) == {1, 2, 3, 4}, splits
    assert ops.tc.lib.gb_gemm_tc_tall(256, 4096, 4096) == 0 and ops.tc.lib.gb_gemm_tc_tall(4096, 4096, 4096) == 0


def test_the_rotating_product_goes_where_it_is_faster(ops):
    """Its epilogue weighs more in these blocks than in the tiles that it would take otherwise, 320 wide ones among them."""
    takes = lambda T, N, K, hd: ops.tc.lib.gb_gemm_tc_tall_rotating(T, N, K, hd) > 0
    assert all(takes(*c) for c in [(257, 1536, 2048, 64), (1793, 2560, 2048, 64), (2400, 2560, 2048, 64), (1221, 6144, 4096, 128)])
    others = [(2048, 2560, 2048, 64), (2300, 2560, 2048, 64), (1511, 6144, 4096, 128), (3500, 1536, 2048, 64), (3500, 1536, 2048, 128),
              (2600, 3072, 3072, 128)]
    assert not any(takes(*c) for c in others) and all(ops.tc.lib.gb_gemm_tc_tall(*c[:3]) > 0 for c in others)


# 32-bit sums of K products of either sign: the order moves them by some units of 2^-24 times sqrt(K)
@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_stored(ops, M, N, K, dtype):
    a, w, want = operands(M, N, K)
    out = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
    ops.linear(a, w, out=out)
    close(out, want.cpu(), dtype, "stored", tol=3e-5 if dtype == torch.float32 else None)


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("alpha", [1.0, 0.37])
def test_added(ops, M, N, K, alpha):
    a, w, want = operands(M, N, K, seed=3)
    out = rnd(M, N, seed=9).cuda()
    want = out + alpha * want
    ops.linear(a, w, out=out, accumulate=True, alpha=alpha)
    close(out, want.cpu(), torch.float32, "added", tol=3e-5)


def test_the_same_bits_every_time(ops):
    a, w, _ = operands(333, 4096, 14336, seed=5)
    assert ops.tc.lib.gb_gemm_tc_tall(333, 4096, 14336) > 1
    outs = [torch.empty(333, 4096, device="cuda") for _ in range(3)]
    for o in outs:
        ops.linear(a, w, out=o)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


# one part and two, each split
@pytest.mark.parametrize("M,N,K", [(300, 288, 2040), (270, 2500, 4104), (511, 2048, 5632), (1221, 4096, 2048)])
@pytest.mark.parametrize("kind", ["relu2", "tanh", "gelu", "xielu"])
def test_stored_through_an_activation(ops, M, N, K, kind):
    from tests.plain.cpu_ops import CpuOps
    assert ops.tc.lib.gb_gemm_tc_tall(M, N, K) > 0
    a, w, want = operands(M, N, K, seed=17)
    out = torch.full((M + 1, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    want, ref = want.cpu(), torch.empty(M, N)
    if kind == "xielu":
        assert ops.tc.linear_xielu(a, w, out[:M], 0.8, 1.3)
        CpuOps().xielu(want, ref, 0.8, 1.3)
    else:
        assert ops.tc.linear_act(a, w, out[:M], kind)
        ref = {"relu2": torch.relu(want) ** 2, "tanh": torch.tanh(want), "gelu": torch.nn.functional.gelu(want)}[kind]
    ops.tc.check_errors()
    close(out[:M], ref, torch.bfloat16, kind)
    assert out[M].isnan().all(), "a store beyond the tokens"


@pytest.mark.parametrize("T,Hq,Hkv,hd,d", [(448, 32, 8, 128, 4096), (300, 4, 2, 64, 4096), (513, 6, 1, 32, 4096), (1030, 12, 2, 16, 4096)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_rotated_into_pages(ops, T, Hq, Hkv, hd, d, interleaved):
    from garuda_b200.engine.batch import Workspace
    from garuda_b200.parts.rotary import RotaryParams
    from tests.plain.cpu_ops import CpuOps
    N, page = (Hq + 2 * Hkv) * hd, 8
    assert ops.tc.lib.gb_gemm_tc_tall_rotating(T, N, d, hd) > 0

    class Ctx:
        ws = Workspace("cuda:0")

    h, w, _ = operands(T, N, d, seed=7)
    h, w = h.cpu(), w.cpu()
    req = torch.tensor([i % 3 for i in range(T)], dtype=torch.int32).sort().values
    positions = torch.cat([s + torch.arange(int((req == r).sum())) for r, s in enumerate((0, 37, 100))]).to(torch.int32)
    width = int(positions.max()) // page + 2
    pages = torch.randperm(3 * width, generator=torch.Generator().manual_seed(T)).int().view(3, width)
    for rotary in (RotaryParams(10000.0, hd, interleaved), None):
        want = [torch.zeros(T, Hq, hd), torch.zeros(3 * width, Hkv, page, hd), torch.zeros(3 * width, Hkv, page, hd)]
        CpuOps().qkv_rope_append(None, h, w, *want, positions, req, pages, Hq, Hkv, hd, rotary, page)
        got = [torch.zeros_like(t, dtype=torch.bfloat16, device="cuda") for t in want]
        ops.qkv_rope_append(Ctx, h.cuda(), w.cuda(), *got, positions.cuda(), req.cuda(), pages.cuda(), Hq, Hkv, hd, rotary, page)
        for a, b, what in zip(got, want, "qkv"):
            close(a, b, torch.bfloat16, what)


@pytest.mark.parametrize("M,d,K", [(300, 2048, 5632), (1221, 4096, 2048), (333, 1000, 2048)])
def test_norm_folded_in(ops, M, d, K):
    from garuda_b200.engine.batch import StepContext, Workspace
    from garuda_b200.parts.norm import RMSNorm
    assert ops.tc.lib.gb_gemm_tc_tall(M, d, K) > 0
    a, w, want = operands(M, d, K, seed=11)
    x = (rnd(M, d, seed=12) * (1 + torch.arange(M) % 5).float()[:, None]).cuda()      # a token's sums are not another's
    gamma = (1 + 0.3 * rnd(d, seed=13)).bfloat16().cuda()
    norm = RMSNorm(d, 1e-3)
    norm.load({"weight": gamma}, ops, torch.bfloat16)
    ctx = StepContext(batch=None, ws=Workspace("cuda:0"), ops=ops, dtype=torch.bfloat16)
    res = x.clone()
    pending = ops.linear(a, w, res, accumulate=True, ctx=ctx, emit_norm=norm)
    want = x + want
    close(res, want.cpu(), torch.float32, "residual", tol=3e-5)
    close(pending.values, (want * gamma.float()).cpu(), torch.bfloat16, "x * weight")
    torch.testing.assert_close(pending.sums.sum(0), (want ** 2).sum(1), rtol=1e-4, atol=1e-6)
    # and products behind it, which scale their results by 1/rms
    v = (rnd(4096, d, seed=14) * d ** -0.5).bfloat16().cuda()
    out = torch.empty(M, 4096 // 2, dtype=torch.bfloat16, device="cuda")
    ops.linear_swiglu(ctx, pending, ops.pack_gate_up(v[:2048], v[2048:]), out)
    h = want * torch.rsqrt((want ** 2).mean(1, keepdim=True) + 1e-3) * gamma.float()
    g, u = h @ v[:2048].float().T, h @ v[2048:].float().T
    close(out, (torch.nn.functional.silu(g) * u).cpu(), torch.bfloat16, "gate/up behind it")
    ops.tc.check_errors()


@pytest.mark.parametrize("M,N,K", [(333, 4096, 14336), (2048, 2048, 2048), (8, 2048, 2048)])
def test_sums_of_another_size_are_refused(ops, M, N, K):
    """The rows of the sums for the norm behind follow from the kernel that is chosen: room for another number is an error, not a write beyond it."""
    from garuda_b200.kernels.ops import KernelError, PendingNorm
    rows = ops.tc.norm_tiles(M, N, K)
    a, w, _ = operands(M, N, K)
    for n in (rows - 1, rows + 1):
        out = torch.zeros(M, N, device="cuda")
        pending = PendingNorm(torch.zeros(M, N, dtype=torch.bfloat16, device="cuda"), torch.zeros(rows + 1, M, device="cuda")[:n],
                              torch.ones(N, device="cuda"), 1e-5, None, out)
        with pytest.raises(KernelError, match="rows of sums"):
            ops.tc.linear(a, w, out, True, emit=pending)
        assert not out.any() and not pending.sums.any()


# split in one, two and four; one block of tokens and several
@pytest.mark.parametrize("T,Hq,Hkv,hd,d", [(448, 32, 8, 128, 4096), (300, 4, 2, 64, 4096), (1030, 12, 2, 16, 4096), (900, 32, 8, 128, 4096)])
def test_rotated_behind_a_folded_norm(ops, T, Hq, Hkv, hd, d):
    """Each token at a scale of its own, which the norm takes out: the factors must be the tokens' own."""
    from garuda_b200.engine.batch import StepContext, Workspace
    from garuda_b200.parts.norm import RMSNorm
    from garuda_b200.parts.rotary import RotaryParams
    from tests.plain.cpu_ops import CpuOps
    N, page = (Hq + 2 * Hkv) * hd, 8
    assert ops.tc.lib.gb_gemm_tc_tall_rotating(T, N, d, hd) > 0
    g = torch.Generator(device="cuda").manual_seed(T)
    a, w_o = (torch.randn(T, 128, generator=g, device="cuda") * 0.5).bfloat16(), (torch.randn(d, 128, generator=g, device="cuda") * 0.1).bfloat16()
    norm = RMSNorm(d, 1e-3)
    norm.load({"weight": (1 + 0.3 * torch.randn(d, generator=g, device="cuda")).bfloat16()}, ops, torch.bfloat16)
    ctx = StepContext(batch=None, ws=Workspace("cuda:0"), ops=ops, dtype=torch.bfloat16)
    res = torch.randn(T, d, generator=g, device="cuda") * (1 + torch.arange(T, device="cuda") % 5)[:, None]
    pending = ops.linear(a, w_o, res, accumulate=True, ctx=ctx, emit_norm=norm)
    assert pending is not None
    h = pending.values.float() * torch.rsqrt((res ** 2).mean(1, keepdim=True) + 1e-3)      # (32-bit rows in the reference)
    w = (torch.randn(N, d, generator=g, device="cuda") * d ** -0.5).bfloat16()
    req = torch.zeros(T, dtype=torch.int32)
    positions, width = torch.arange(T, dtype=torch.int32) + 19, (T + 19) // page + 1
    pages = torch.randperm(width, generator=torch.Generator().manual_seed(T)).int().view(1, width)
    rotary = RotaryParams(10000.0, hd, False)
    want = [torch.zeros(T, Hq, hd), torch.zeros(width, Hkv, page, hd), torch.zeros(width, Hkv, page, hd)]
    CpuOps().qkv_rope_append(None, h.cpu(), w.float().cpu(), *want, positions, req, pages, Hq, Hkv, hd, rotary, page)
    got = [torch.zeros_like(t, dtype=torch.bfloat16, device="cuda") for t in want]
    ops.qkv_rope_append(ctx, pending, w, *got, positions.cuda(), req.cuda(), pages.cuda(), Hq, Hkv, hd, rotary, page)
    ops.tc.check_errors()
    for x, y, what in zip(got, want, "qkv"):
        close(x, y, torch.bfloat16, what)

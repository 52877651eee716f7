"""The gated product of some hundreds of tokens on tiles of up to 512 tokens: parts of each width, a last tile without a second
group of features, features that are no multiple of a group or of eight, pairs with several tiles, each activation, a folded norm."""
import pytest
import torch

from tests.gpu_helpers import close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from garuda_b200.kernels.ops import CudaOps
    return CudaOps("cuda:0")


# tokens: the fewest and most of the parts of 160, 192, 224 and 256 that the rule lets through; 112 and 113 tiles on 74 pairs
@pytest.mark.parametrize("T,F,K,kind", [
    (257, 14336, 4096, "silu"), (320, 14330, 4104, "silu"), (321, 14272, 4096, "gelu_tanh"), (384, 14336, 4096, "silu"),
    (385, 14400, 4096, "clamped_swish"), (448, 14336, 5000, "silu"), (449, 14332, 8192, "silu"), (512, 6149, 8192, "gelu_tanh"), (512, 6144, 8192, "silu")])
def test_gated_product(ops, T, F, K, kind):
    g = torch.Generator(device="cuda").manual_seed(T + F)
    h = (torch.randn(T, K, generator=g, device="cuda") * 0.5).bfloat16()
    gate, up = ((torch.randn(F, K, generator=g, device="cuda") * 0.05).bfloat16() for _ in range(2))
    room = torch.full((T + 1, F), float("nan"), dtype=torch.bfloat16, device="cuda")
    room[T] = 9.0
    packed = ops.pack_gate_up(gate, up)
    assert ops.tc.lib.gb_gemm_tc_wide(T, packed.shape[0], K) == 1, "the sizes are for the wide tiles"
    assert ops.tc.linear_swiglu(h, packed, room[:T], kind=ops.GATE_ACTS[kind], limit=3.0)
    ops.tc.check_errors()
    a, u = h.double() @ gate.double().T, h.double() @ up.double().T
    if kind == "clamped_swish":
        a, u = a.clamp(max=3.0), u.clamp(-3.0, 3.0)
        want = a * torch.sigmoid(1.702 * a) * (u + 1)
    else:
        want = (torch.nn.functional.silu(a) if kind == "silu" else torch.nn.functional.gelu(a, approximate="tanh")) * u
    close(room[:T], want.cpu(), torch.bfloat16, "gated product", tol=2 ** -8)      # half of bfloat16's last place, of the largest
    assert (room[T] == 9.0).all(), "a store beyond the tokens"


@pytest.mark.parametrize("T", [257, 400, 448])
def test_behind_a_folded_norm(ops, T):
    """Each token at a scale of its own, taken out by the norm: the factors must be the tokens' own."""
    from garuda_b200.engine.batch import StepContext, Workspace
    from garuda_b200.parts.norm import RMSNorm
    d, K, F = 4096, 128, 14336
    g = torch.Generator(device="cuda").manual_seed(T)
    a, w_o = (torch.randn(T, K, generator=g, device="cuda") * 0.5).bfloat16(), (torch.randn(d, K, generator=g, device="cuda") * 0.1).bfloat16()
    norm = RMSNorm(d, 1e-3)
    norm.load({"weight": torch.ones(d, dtype=torch.bfloat16, device="cuda")}, ops, torch.bfloat16)
    ctx = StepContext(batch=None, ws=Workspace("cuda:0"), ops=ops, dtype=torch.bfloat16)
    res = torch.randn(T, d, generator=g, device="cuda") * (1 + torch.arange(T, device="cuda") % 5)[:, None]
    pending = ops.linear(a, w_o, res, accumulate=True, ctx=ctx, emit_norm=norm)
    assert pending is not None
    h = pending.values.double() * torch.rsqrt((res.double() ** 2).mean(1, keepdim=True) + 1e-3)
    gate, up = ((torch.randn(F, d, generator=g, device="cuda") * 0.02).bfloat16() for _ in range(2))
    out = torch.full((T, F), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.linear_swiglu(ctx, pending, ops.pack_gate_up(gate, up), out)
    ops.tc.check_errors()
    close(out, (torch.nn.functional.silu(h @ gate.double().T) * (h @ up.double().T)).cpu(), torch.bfloat16, "behind a norm", tol=2 ** -8)


@pytest.mark.parametrize("kind", ["silu", "gelu_tanh", "clamped_swish"])
def test_the_tiles_do_not_show(ops, kind):
    """A token's result is the same bits in a step of 400 tokens (wide tiles) as in one of 600 (the other tiles), gates up to
    70 on both sides among them (below -87 the two may differ in a last place of results below 1e-35)."""
    F, K, T = 14336, 4096, 400
    g = torch.Generator(device="cuda").manual_seed(7)
    h = (torch.randn(600, K, generator=g, device="cuda") * 0.5).bfloat16()
    h[::7] *= 8.0
    w = ops.pack_gate_up(*((torch.randn(F, K, generator=g, device="cuda") * 0.05).bfloat16() for _ in range(2)))
    outs = [torch.zeros(n, F, dtype=torch.bfloat16, device="cuda") for n in (T, 600)]
    for n, out in zip((T, 600), outs):
        assert ops.tc.linear_swiglu(h[:n], w, out, kind=ops.GATE_ACTS[kind], limit=50.0)
    ops.tc.check_errors()
    assert torch.equal(outs[0], outs[1][:T])

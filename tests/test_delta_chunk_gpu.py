"""The delta rules walked by chunks of 32 tokens (bfloat16 runs, requests of many tokens) against the
plain references, which walk token by token: chunks that are full, one short and one over, requests
below the line beside requests above it, a state that is carried over, padding rows, decays so strong
that a chunk's product of them underflows, rows that are column ranges of wider ones."""
import pytest
import torch

from tests.gpu_helpers import batches, close, rnd, step_batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from garuda_b200.kernels.ops import CudaOps
    from tests.plain.cpu_ops import CpuOps
    return CudaOps("cuda:0"), CpuOps()


CUT = 48
STEPS = [(CUT - 1, CUT, 97), (1, 64, 5), (CUT, 1, 1), (65, 63, 50)]


def step(lens, slots):
    return step_batch(lens, [0] * len(lens), slots, 16)[0]


@pytest.mark.parametrize("H,G,dim,vdim,taps,per_head,strong", [
    (2, 2, 64, 64, 4, False, False), (4, 2, 128, 128, 4, True, False), (1, 1, 128, 32, 1, False, True), (3, 1, 64, 160, 3, True, True),
    (40, 20, 64, 96, 2, False, False), (2, 1, 128, 256, 4, False, False)])
def test_gated_rule(ops, H, G, dim, vdim, taps, per_head, strong):
    cuda, cpu = ops
    assert cuda.DELTA_CHUNK_CUT == CUT
    C, n_decay = 2 * G * dim + H * vdim, H if per_head else H * dim
    n_state = H * dim * vdim
    conv_w, a_log = rnd(C, taps, scale=0.5), rnd(H, scale=0.5, seed=1) + (3.0 if strong else 0.0)
    dt_bias, norm_w = rnd(n_decay, seed=2) - (0.0 if strong else 3.0), rnd(vdim, seed=3) + 1.0
    state_g, state_r = torch.zeros(5, n_state + (taps - 1) * C, device="cuda"), torch.zeros(5, n_state + (taps - 1) * C)
    state_g[4] = float("nan")                           # a slot nobody uses
    for k, lens in enumerate(STEPS):
        T = sum(lens)
        ctx_g, ctx_r = batches(step(lens, [3, 0, 2]))
        wide = rnd(T, 3 + C + H + n_decay + H * vdim + 5, scale=1.5, seed=10 + k)
        first, second = 3 + C + H, 3 + C + H + n_decay + H * vdim
        out, ref = torch.zeros(T, H * vdim, dtype=torch.bfloat16, device="cuda"), torch.zeros(T, H * vdim, dtype=torch.bfloat16)
        before = cuda.launches
        for o, c, row, st, to, y in ((cuda, ctx_g, wide.cuda(), state_g, lambda t: t.cuda(), out), (cpu, ctx_r, wide, state_r, lambda t: t, ref)):
            o.delta_rule(c, row[:, 3:first], row[:, first:second], to(conv_w), to(a_log), to(dt_bias), to(norm_w), 1e-5, st, H, G, dim, vdim,
                         taps, y, decay_per_head=per_head, gate="silu" if per_head else "sigmoid")
        assert cuda.launches - before == 2 + 2 * (min(lens) < CUT) + 2, "the step's chunked kernels, and the others beside them"
        close(out, ref, torch.bfloat16, f"step {k}: outputs")
        # sums of at most 256 terms of 32-bit, a hundred tokens deep: the two orders differ by parts in a million
        close(state_g[:4], state_r[:4], torch.float32, f"step {k}: state", tol=2e-5)


@pytest.mark.parametrize("H,dim,vdim,strong", [(2, 64, 64, False), (3, 128, 128, False), (1, 64, 32, True), (50, 64, 96, False), (2, 128, 160, True)])
def test_general_rule(ops, H, dim, vdim, strong):
    cuda, cpu = ops
    HD, HV = H * dim, H * vdim
    cols = (3, 3 + HD, 3 + 2 * HD, 3 + 2 * HD + HV, 3 + 3 * HD + HV)
    w0, a0, norm_w = rnd(HD, scale=1.5, seed=1) - 2.0, rnd(HD, seed=2), rnd(HV, seed=3) + 1.0
    state_g, state_r = torch.zeros(5, HD * vdim, device="cuda"), torch.zeros(5, HD * vdim)
    state_g[1] = float("nan")
    # from how many tokens on a request is walked by chunks, and where there are shorter ones beside it
    cut, mixed = (128, 160) if dim == 64 else (CUT, 100)
    assert cuda.GENERAL_CHUNK_CUTS[dim > 64] == (cut, mixed)
    for k, lens in enumerate(STEPS + [(cut - 1, 1, mixed - 1), (mixed, 1, cut - 1), (1, cut, 256)] + [(cut + 1, 10, cut - 3)] * (dim == 128)):
        T = sum(lens)
        ctx_g, ctx_r = batches(step(lens, [3, 0, 2]))
        proj, zdec = rnd(T, cols[4] + HV + 6, scale=1.5, seed=10 + k), rnd(T, HD + 2, scale=2.0, seed=20 + k)
        out, ref = torch.zeros(T, HV, dtype=torch.bfloat16, device="cuda"), torch.zeros(T, HV, dtype=torch.bfloat16)
        for o, c, st, to, y in ((cuda, ctx_g, state_g, lambda t: t.cuda(), out), (cpu, ctx_r, state_r, lambda t: t, ref)):
            o.general_delta(c, to(proj), cols, to(zdec)[:, :HD], to(w0), to(a0), 20.0 if strong else 0.6, to(norm_w), 1e-5, st, H, dim, vdim, y)
        walks = max(lens) >= cut and (min(lens) >= cut or max(lens) >= mixed or T >= 256)
        assert ("delta_blocks" in ctx_g.ws._bufs) == walks, lens
        close(out, ref, torch.bfloat16, f"step {k}: outputs")
        keep = [0, 2, 3, 4]
        close(state_g[keep], state_r[keep], torch.float32, f"step {k}: state", tol=2e-5)


@pytest.mark.parametrize("counted", [True, False])
@pytest.mark.parametrize("lens", [(CUT + 52,) + (1,) * 40, (3, 0, 107, 1, 0, 64) + (2,) * 40 + (CUT, 1), (0, CUT, 0)])
def test_scratch_is_for_the_requests_that_are_walked(ops, lens, counted):
    """Single tokens (and requests without any) beside a few long stretches: no room for those that are not walked, whether the batch
    brings its lengths on the host or not; more than a warp's requests in front of one that is walked."""
    cuda, cpu = ops
    H, dim, vdim, taps, R, T = 2, 64, 32, 2, len(lens), sum(lens)
    C, long = 2 * H * dim + H * vdim, sum(n >= CUT for n in lens)
    b = step(list(lens), list(range(R))[::-1])
    if counted:
        b.host = {"cu_q": b.cu_q.numpy()}
    ctx_g, ctx_r = batches(b)
    room = T // 32 + (long if counted else min(R, T // CUT))
    args = [rnd(T, C + H, scale=1.5), rnd(T, H + H * vdim, seed=1), rnd(C, taps, seed=2), rnd(H, seed=3), rnd(H, seed=4), rnd(vdim, seed=5)]
    state = rnd(R, H * dim * vdim + (taps - 1) * C, seed=6)
    got, want = state.cuda(), state.clone()
    out, ref = torch.zeros(T, H * vdim, dtype=torch.bfloat16, device="cuda"), torch.zeros(T, H * vdim, dtype=torch.bfloat16)
    cuda.delta_rule(ctx_g, *(t.cuda() for t in args), 1e-5, got, H, H, dim, vdim, taps, out, decay_per_head=True)
    cpu.delta_rule(ctx_r, *args, 1e-5, want, H, H, dim, vdim, taps, ref, decay_per_head=True)
    close(out, ref, torch.bfloat16, "gated rule: outputs")
    close(got, want, torch.float32, "gated rule: state", tol=2e-5)
    chunk = 96 * dim + dim + 64 * vdim               # W, Q and K1; the chunk's decay; VP and OP
    assert ctx_g.ws._bufs["delta_blocks"].numel() <= room * H * chunk * 4 + 256
    ctx_g, ctx_r = batches(b)
    dim = 128                                        # (the generalized rule of 64 channels walks longer stretches only)
    HD, HV = H * dim, H * vdim
    cols = (0, HD, 2 * HD, 2 * HD + HV, 3 * HD + HV)
    args = [rnd(T, cols[4] + HV, scale=1.5, seed=7), cols, rnd(T, HD, seed=8), rnd(HD, seed=9), rnd(HD, seed=10), 0.6, rnd(HV, seed=11)]
    to = lambda v: v.cuda() if torch.is_tensor(v) else v
    state = rnd(R, HD * vdim, seed=6)
    got, want = state.cuda(), state.clone()
    cuda.general_delta(ctx_g, *map(to, args), 1e-5, got, H, dim, vdim, out)
    cpu.general_delta(ctx_r, *args, 1e-5, want, H, dim, vdim, ref)
    close(out, ref, torch.bfloat16, "general rule: outputs")
    close(got, want, torch.float32, "general rule: state", tol=2e-5)
    chunk = 128 * dim + dim + 96 * vdim              # K2 and V beside them
    walks = T >= 256 or max(lens) >= 100 or min(lens) >= CUT
    assert ctx_g.ws._bufs["delta_blocks"].numel() <= room * H * chunk * 4 + 256 if walks else "delta_blocks" not in ctx_g.ws._bufs


def test_padding_rows_touch_no_state(ops):
    cuda, _ = ops
    H, dim, vdim, taps = 2, 64, 32, 4
    C = 2 * H * dim + H * vdim
    state = rnd(3, H * dim * vdim + (taps - 1) * C).cuda()
    before = state.clone()
    ctx, _ = batches(step([CUT + 5, 70], [-1, -1]))
    out = torch.zeros(CUT + 75, H * vdim, dtype=torch.bfloat16, device="cuda")
    cuda.delta_rule(ctx, rnd(CUT + 75, C + H).cuda(), rnd(CUT + 75, H + H * vdim).cuda(), rnd(C, taps).cuda(), rnd(H).cuda(), rnd(H).cuda(),
                    rnd(vdim).cuda(), 1e-5, state, H, H, dim, vdim, taps, out, decay_per_head=True)
    assert torch.equal(state, before) and torch.isfinite(out.float()).all()


def test_a_value_that_is_not_a_number_leaves_the_tokens_in_front_of_it_alone(ops):
    cuda, _ = ops
    H, dim, vdim, taps, T, bad = 2, 64, 64, 4, 100, 45
    C = 2 * H * dim + H * vdim
    proj, second = rnd(T, C + H).cuda(), rnd(T, H + H * vdim, seed=1).cuda()
    w = [t.cuda() for t in (rnd(C, taps, seed=2), rnd(H, seed=3), rnd(H, seed=4), rnd(vdim, seed=5))]
    outs = []
    for spoil in (False, True):
        p = proj.clone()
        if spoil:
            p[bad] = float("nan")
        ctx, _ = batches(step([T], [0]))
        outs.append(torch.zeros(T, H * vdim, dtype=torch.bfloat16, device="cuda"))
        state = torch.zeros(1, H * dim * vdim + (taps - 1) * C, device="cuda")
        cuda.delta_rule(ctx, p, second, *w, 1e-5, state, H, H, dim, vdim, taps, outs[-1], decay_per_head=True)
    assert torch.equal(outs[0][:bad], outs[1][:bad]) and torch.isnan(outs[1][bad:].float()).all()


@pytest.mark.parametrize("taps", [1, 2, 3, 4])
def test_a_query_that_is_not_a_number_reaches_as_far_as_the_taps(ops, taps):
    cuda, _ = ops
    H, dim, vdim, T, bad = 2, 64, 64, 100, 45
    C = 2 * H * dim + H * vdim
    proj, second = rnd(T, C + H).cuda(), rnd(T, H + H * vdim, seed=1).cuda()
    w = [t.cuda() for t in (rnd(C, taps, seed=2), rnd(H, seed=3), rnd(H, seed=4), rnd(vdim, seed=5))]
    outs, states = [], []
    for spoil in (0.0, float("inf"), float("nan")):
        p = proj.clone()
        p[bad, :H * dim] += spoil                       # the queries' inputs alone: nothing of it may stay in the state
        ctx, _ = batches(step([T], [0]))
        outs.append(torch.zeros(T, H * vdim, dtype=torch.bfloat16, device="cuda"))
        states.append(torch.zeros(1, H * dim * vdim + (taps - 1) * C, device="cuda"))
        cuda.delta_rule(ctx, p, second, *w, 1e-5, states[-1], H, H, dim, vdim, taps, outs[-1], decay_per_head=True)
    for out, state in zip(outs[1:], states[1:]):
        hit = torch.isnan(out.float()).any(1)
        assert hit[bad:bad + taps].all() and hit.sum() == taps and torch.equal(out[~hit], outs[0][~hit])
        assert torch.equal(state[:, :H * dim * vdim], states[0][:, :H * dim * vdim])


def test_a_32_bit_run_is_walked_token_by_token(ops):
    """There the numbers do not depend on how a prompt was cut."""
    cuda, _ = ops
    H, dim, vdim, taps, T = 2, 64, 64, 3, 130
    C = 2 * H * dim + H * vdim
    proj, second = rnd(T, C + H).cuda(), rnd(T, H + H * vdim, seed=1).cuda()
    w = [t.cuda() for t in (rnd(C, taps, seed=2), rnd(H, seed=3), rnd(H, seed=4), rnd(vdim, seed=5))]
    got = []
    for cuts in ([T], [61, 69]):
        state, at, outs = torch.zeros(1, H * dim * vdim + (taps - 1) * C, device="cuda"), 0, []
        for n in cuts:
            ctx, _ = batches(step([n], [0]))
            outs.append(torch.zeros(n, H * vdim, device="cuda"))
            cuda.delta_rule(ctx, proj[at:at + n], second[at:at + n], *w, 1e-5, state, H, H, dim, vdim, taps, outs[-1], decay_per_head=True)
            at += n
        got.append((torch.cat(outs), state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def test_a_cut_where_a_chunk_ends_moves_no_bit(ops):
    cuda, _ = ops
    H, dim, vdim, taps, T = 2, 128, 64, 4, 192
    C = 2 * H * dim + H * vdim
    proj, second = rnd(T, C + H).cuda(), rnd(T, H * dim + H * vdim, seed=1).cuda()
    w = [t.cuda() for t in (rnd(C, taps, seed=2), rnd(H, seed=3), rnd(H * dim, seed=4), rnd(vdim, seed=5))]
    got = []
    for cuts in ([T], [96, 96], [128, 64]):
        state, at, outs = torch.zeros(1, H * dim * vdim + (taps - 1) * C, device="cuda"), 0, []
        for n in cuts:
            ctx, _ = batches(step([n], [0]))
            outs.append(torch.zeros(n, H * vdim, dtype=torch.bfloat16, device="cuda"))
            cuda.delta_rule(ctx, proj[at:at + n], second[at:at + n], *w, 1e-5, state, H, H, dim, vdim, taps, outs[-1])
            at += n
        got.append((torch.cat(outs), state))
    assert all(torch.equal(a, b) for other in got[1:] for a, b in zip(got[0], other))


def _gated64(proj, second, conv_w, a_log, dt_bias, H, G, dim, vdim, taps, per_head):
    T, C, dev = proj.shape[0], 2 * G * dim + H * vdim, proj.device
    x = torch.cat([torch.zeros(taps - 1, C, device=dev, dtype=torch.float64), proj[:, :C].double()])
    a = torch.nn.functional.silu(sum(x[i:i + T] * conv_w.double()[:, i] for i in range(taps)))
    q, k, v = (t.view(T, -1, n) for t, n in zip(a.split([G * dim, G * dim, H * vdim], 1), (dim, dim, vdim)))
    q, k = ((t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1) for t in (q, k))
    beta, rate = torch.sigmoid(proj[:, C:].double()), torch.exp(a_log.double())
    step = torch.nn.functional.softplus(second[:, :dt_bias.numel()].double() + dt_bias.double()).view(T, H, -1)
    g = torch.exp(-rate[:, None] * step)
    S, o = torch.zeros(H, dim, vdim, dtype=torch.float64, device=dev), torch.empty(T, H, vdim, dtype=torch.float64, device=dev)
    for t in range(T):
        S *= g[t][:, :, None]
        S += k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t])))[:, None, :]
        o[t] = torch.einsum("hdv,hd->hv", S, q[t]) * dim ** -0.5
    return o, S


def _general64(proj, cols, zdec, w0, a0, scale, H, dim, vdim):
    T, dev = proj.shape[0], proj.device
    r, k, v, a = (proj[:, c:c + n].double() for c, n in zip(cols, (H * dim, H * dim, H * vdim, H * dim)))
    a, w = torch.sigmoid(a + a0.double()).view(T, H, dim), torch.exp(-scale * torch.sigmoid(zdec.double() + w0.double())).view(T, H, dim)
    r, k, v = r.view(T, H, dim), k.view(T, H, dim), v.view(T, H, vdim)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    S, o = torch.zeros(H, dim, vdim, dtype=torch.float64, device=dev), torch.empty(T, H, vdim, dtype=torch.float64, device=dev)
    for t in range(T):
        S = w[t][:, :, None] * S - (a[t] * u[t])[:, :, None] * torch.einsum("hdv,hd->hv", S, u[t])[:, None, :] + k[t][:, :, None] * v[t][:, None, :]
        o[t] = torch.einsum("hdv,hd->hv", S, r[t])
    return o, S


@pytest.mark.parametrize("rule,dim,decay", [("channel", 128, -3.0), ("channel", 128, -8.0), ("head", 128, -3.0), ("head", 128, -8.0), ("head", 64, -5.0),
                                            ("general", 64, -3.0), ("general", 64, -8.0), ("general", 128, -3.0), ("general", 128, -8.0)])
def test_as_near_64_bits_as_the_walk_token_by_token(ops, rule, dim, decay):
    """2,048 tokens, decays that forget in a few tokens to some thousand: the read-outs and the state may be no further off than those of the
    32-bit walk (what a 32-bit run takes). The two round at different places, so their errors are two draws of one size: 1.2 of it."""
    cuda, _ = ops
    H, G, T, taps, vdim = 4, 2, 2048, 4, dim
    g = torch.Generator(device="cuda").manual_seed(dim)
    draw = lambda *s, std=1.0, mean=0.0: torch.randn(*s, generator=g, device="cuda") * std + mean
    if rule == "general":
        HD = H * dim
        cols = (0, HD, 2 * HD, 3 * HD, 4 * HD)
        args = [draw(T, 5 * HD), cols, draw(T, HD), draw(HD, mean=decay), draw(HD), 0.6]
        ref, width = _general64(*args, H, dim, vdim), HD * vdim
    else:
        C, n_decay = 2 * G * dim + H * vdim, H if rule == "head" else H * dim
        args = [draw(T, C + H), draw(T, n_decay + H * vdim), draw(C, taps, std=0.5), draw(H, std=0.3), draw(n_decay, std=0.3, mean=decay)]
        ref, width = _gated64(*args, H, G, dim, vdim, taps, rule == "head"), H * dim * vdim + (taps - 1) * C
    off = []
    for dt in (torch.float32, torch.bfloat16):
        ctx, _ = batches(step([T], [0]))
        state, out = torch.zeros(1, width, device="cuda"), torch.zeros(T, H * vdim, dtype=dt, device="cuda")
        if rule == "general":
            cuda.general_delta(ctx, *args, torch.ones(H * vdim, device="cuda"), 1e-5, state, H, dim, vdim, out)
        else:
            cuda.delta_rule(ctx, *args, torch.ones(vdim, device="cuda"), 1e-5, state, H, G, dim, vdim, taps, out, decay_per_head=rule == "head")
        assert ("delta_blocks" in ctx.ws._bufs) == (dt == torch.bfloat16)
        o = ctx.ws._views["gdelta_o" if rule == "general" else "delta_o"][2]
        off.append([((x.double().flatten() - y.flatten()).norm() / y.norm()).item() for x, y in zip((o, state[:, :H * dim * vdim]), ref)])
    assert all(chunk <= 1.2 * token for token, chunk in zip(*off)), f"read-outs, state: token by token {off[0]}, by chunks {off[1]}"


@pytest.mark.parametrize("rule,dim,decay,most", [
    # decays that keep thousands of tokens: the chunks hold what a decay lacks of one, the walk the decay rounded to 24 bits
    ("channel", 128, -8.0, 0.4), ("head", 64, -8.0, 0.4), ("general", 64, -8.0, 0.4), ("general", 128, -8.0, 0.4),
    # decays that keep some tens of tokens: sums and triangular systems of 32 tokens may not be rounded further off than the walk's steps (the mean
    # of six draws of 262,144 numbers: two kernels of one precision differ by a hundredth)
    ("channel", 128, -3.0, 1.01), ("head", 128, -3.0, 1.01)])
def test_readouts_no_further_from_64_bits_than_the_walk_token_by_token(ops, rule, dim, decay, most):
    cuda, _ = ops
    H, G, T, taps = 4, 2, 512, 4
    off = torch.zeros(2)
    for seed in range(6):
        g = torch.Generator(device="cuda").manual_seed(100 * dim + seed)
        draw = lambda *s, std=1.0, mean=0.0: torch.randn(*s, generator=g, device="cuda") * std + mean
        if rule == "general":
            HD = H * dim
            cols = (0, HD, 2 * HD, 3 * HD, 4 * HD)
            args, width = [draw(T, 5 * HD), cols, draw(T, HD), draw(HD, mean=decay), draw(HD), 0.6], HD * dim
            ref = _general64(*args, H, dim, dim)[0]
        else:
            C, n_decay, width = (2 * G + H) * dim, H if rule == "head" else H * dim, H * dim * dim + (taps - 1) * (2 * G + H) * dim
            args = [draw(T, C + H), draw(T, n_decay + H * dim), draw(C, taps, std=0.5), draw(H, std=0.3), draw(n_decay, std=0.3, mean=decay)]
            ref = _gated64(*args, H, G, dim, dim, taps, rule == "head")[0]
        for i, dt in enumerate((torch.float32, torch.bfloat16)):
            ctx, _ = batches(step([T], [0]))
            state, out = torch.zeros(1, width, device="cuda"), torch.zeros(T, H * dim, dtype=dt, device="cuda")
            if rule == "general":
                cuda.general_delta(ctx, *args, torch.ones(H * dim, device="cuda"), 1e-5, state, H, dim, dim, out)
            else:
                cuda.delta_rule(ctx, *args, torch.ones(dim, device="cuda"), 1e-5, state, H, G, dim, dim, taps, out, decay_per_head=rule == "head")
            o = ctx.ws._views["gdelta_o" if rule == "general" else "delta_o"][2]
            off[i] += ((o.double().flatten() - ref.flatten()).norm() / ref.norm()).item()
    assert off[1] <= most * off[0], f"token by token {off[0] / 6:.3e}, by chunks {off[1] / 6:.3e}"


def test_a_state_that_grows(ops):
    """The generalized rule takes any scale: a negative one makes the state grow."""
    cuda, cpu = ops
    H, dim, vdim, T = 2, 64, 64, 150
    HD = H * dim
    cols = (0, HD, 2 * HD, 3 * HD, 4 * HD)
    args = [rnd(T, 5 * HD, scale=0.5), cols, rnd(T, HD, seed=1), rnd(HD, seed=2) - 3.0, rnd(HD, seed=3), -0.2, rnd(HD, seed=4)]
    to = lambda v: v.cuda() if torch.is_tensor(v) else v
    state = rnd(1, HD * vdim, seed=6)
    got, want = state.cuda(), state.clone()
    out, ref = torch.zeros(T, HD, dtype=torch.bfloat16, device="cuda"), torch.zeros(T, HD, dtype=torch.bfloat16)
    ctx_g, ctx_r = batches(step([T], [0]))
    cuda.general_delta(ctx_g, *map(to, args), 1e-5, got, H, dim, vdim, out)
    cpu.general_delta(ctx_r, *args, 1e-5, want, H, dim, vdim, ref)
    assert "delta_blocks" in ctx_g.ws._bufs
    close(out, ref, torch.bfloat16, "outputs")
    close(got, want, torch.float32, "state", tol=2e-5)

"""Capped attention of prompt portions on the tcgen05 kernel against 64-bit attention: each option by itself and together, widths of
64 and 128, scores beyond the cap, windows and stretches whose edges fall inside and between tiles of 64 keys, kept first
positions in the window's own tiles and below them, pages given back, whatever lies where no query reads, single tokens
beside portions."""
import math

import pytest
import torch

from tests.gpu_helpers import close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from garuda_b200.kernels.ops import CudaOps
    return CudaOps("cuda:0")


REQS = [(200, 200), (64, 64), (700, 130), (65, 33), (300, 1), (1000, 3)]


@pytest.mark.parametrize("kd,vd,Hq,Hkv,page,cap,window,keep,sink,far,chunk", [
    (64, 64, 8, 2, 32, 30.0, 150, 4, "one", False, 0), (64, 64, 4, 4, 8, 2.0, 0, 0, "", False, 0), (128, 128, 16, 2, 16, 0.0, 0, 0, "heads", False, 0),
    (64, 64, 32, 1, 64, 0.0, 0, 0, "heads", True, 128), (128, 64, 8, 1, 32, 5.0, 64, 130, "one", True, 0), (64, 128, 2, 1, 16, 0.0, 97, 1, "", False, 0),
    (128, 128, 8, 8, 32, 0.0, 0, 0, "", True, 100)])
def test_prompt_portions(ops, kd, vd, Hq, Hkv, page, cap, window, keep, sink, far, chunk):
    R, T, dev = len(REQS), sum(n for _, n in REQS), "cuda"
    g = torch.Generator(device=dev).manual_seed(kd + vd + page)
    each = [(kv + page - 1) // page for kv, _ in REQS]
    total = sum(each) + 2
    kp = torch.full((total, Hkv, page, kd), float("nan"), dtype=torch.bfloat16, device=dev)      # what nobody wrote
    vp = torch.full((total, Hkv, page, vd), float("nan"), dtype=torch.bfloat16, device=dev)
    order = torch.randperm(total, generator=g, device=dev).int()
    table = torch.full((R, max(each) + 1), -1, dtype=torch.int32, device=dev)
    q = (torch.randn(T, Hq, kd, generator=g, device=dev) * 2.0).bfloat16()
    sinks = torch.randn(Hq, generator=g, device=dev) + 1.0 if sink == "heads" else None
    r1, r2 = (torch.rand(Hq, generator=g, device=dev) + 0.1 for _ in range(2)) if far else (None, None)
    scale, at, t0, ref = kd ** -0.5, 0, 0, torch.empty(T, Hq, vd, dtype=torch.float64, device=dev)
    for r, (kv, n) in enumerate(REQS):
        table[r, :each[r]] = order[at:at + each[r]]
        at += each[r]
        k, v = (torch.randn(kv, Hkv, w, generator=g, device=dev).bfloat16() for w in (kd, vd))
        j = torch.arange(kv, device=dev)
        where = table[r].long()[j // page]
        kp[where, :, j % page], vp[where, :, j % page] = k, v
        i = kv - n + torch.arange(n, device=dev)
        seen = j[None, :] <= i[:, None]
        if chunk:
            seen &= (j // chunk)[None, :] == (i // chunk)[:, None]
        if window:
            seen &= (i[:, None] - j[None, :] < window) | (j[None, :] < keep)
            # pages of which no query of the step reads a key were given back, and what lies in the others may be anything
            unread = ~seen.any(0)
            vp[where[unread], :, (j % page)[unread]] = float("nan")
            for pg in range(each[r]):
                if unread[pg * page:(pg + 1) * page].all():
                    table[r, pg] = -1
        for h in range(Hq):
            s = q[t0:t0 + n, h].double() @ k[:, h // (Hq // Hkv)].double().T * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            if far:
                s = s - r1[h].double() * torch.log1p(r2[h].double() * (i[:, None] - j[None, :]).clamp(min=0))
            e = torch.exp(s - 20.0).masked_fill(~seen, 0.0)
            den = e.sum(-1, keepdim=True) + (math.exp(-20.0) if sink == "one" else 0.0)
            if sinks is not None:
                den = den + torch.exp(sinks[h].double() - 20.0)
            ref[t0:t0 + n, h] = (e / den) @ v[:, h // (Hq // Hkv)].double()
        t0 += n
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    cu = i32([sum(n for _, n in REQS[:r]) for r in range(R + 1)])
    req = torch.repeat_interleave(torch.arange(R, dtype=torch.int32), torch.tensor([n for _, n in REQS])).cuda()
    out = torch.full((T, Hq * vd), float("nan"), dtype=torch.bfloat16, device=dev)
    ops.paged_attention(q, kp, vp, table, cu, i32([kv for kv, _ in REQS]), req, out, scale, window, page, R, max(n for _, n in REQS),
                        max(kv for kv, _ in REQS), softcap=cap, keep_first=keep, sink=sink == "one", sink_values=sinks,
                        distance=(r1, r2) if far else None, chunk=chunk)
    ops.tc.check_errors()
    assert ops.tc._capped[kd, vd].gb_capped_attention_tc_takes(*(t.data_ptr() for t in (q, kp, vp, out)), R, Hq, Hkv, scale, page, total) == 1
    close(out.view(T, Hq, vd), ref.cpu(), torch.bfloat16, "capped attention")


def test_a_score_that_is_not_a_number(ops):
    """Beside scores within the cap and beside one beyond it: the rows that read it are not numbers, the others as if it were not there."""
    Hq, Hkv, hd, page, n, bad, large = 8, 2, 64, 16, 128, 50, 40
    g = torch.Generator(device="cuda").manual_seed(3)
    q, kp, vp = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((n, Hq, hd), (n // page, Hkv, page, hd), (n // page, Hkv, page, hd)))
    table = torch.arange(n // page, dtype=torch.int32, device="cuda")[None]
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    for beyond in (False, True):
        if beyond:
            kp[large // page, :, large % page] *= 100.0
        outs = []
        for k in (kp, kp.clone()):
            if outs:
                k[bad // page, :, bad % page] = float("nan")
            outs.append(torch.zeros(n, Hq * hd, dtype=torch.bfloat16, device="cuda"))
            ops.paged_attention(q, k, vp, table, i32(0, n), i32(n), torch.zeros(n, dtype=torch.int32, device="cuda"), outs[-1], hd ** -0.5, 0, page, 1, n, n,
                                softcap=5.0)
        assert torch.isfinite(outs[0]).all() and torch.equal(outs[0][:bad], outs[1][:bad]) and torch.isnan(outs[1][bad:]).all()


@pytest.mark.parametrize("hd,cap,chunk", [(64, 0.0, 512), (128, 30.0, 0)])
def test_the_largest_weight_is_not_rounded(ops, hd, cap, chunk):
    """Every value is one and two keys have a weight: the result is one, whatever the later key's score is above the earlier one's. Its
    weight, taken against any other score than the largest, would be rounded to bfloat16 and be off by up to a 256th."""
    Hq, Hkv, page, n, late = 16, 2, 32, 300, 70
    kp = torch.zeros(n // page + 1, Hkv, page, hd, dtype=torch.bfloat16, device="cuda")
    vp = torch.ones_like(kp)
    kp[..., 0], kp[0, :, 0, 0], kp[late // page, :, late % page, 0] = -1000.0, 0.0, 1.0
    q = torch.zeros(n, Hq, hd, dtype=torch.bfloat16, device="cuda")
    q[:, :, 0] = torch.linspace(0.1, 5.5, n * Hq, device="cuda").view(n, Hq).bfloat16()
    table = torch.arange(n // page + 1, dtype=torch.int32, device="cuda")[None]
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    out = torch.full((n, Hq * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.paged_attention(q, kp, vp, table, i32(0, n), i32(n), torch.zeros(n, dtype=torch.int32, device="cuda"), out, 1.0, 0, page, 1, n, n, softcap=cap, chunk=chunk)
    ops.tc.check_errors()
    assert torch.equal(out, torch.ones_like(out))


def test_what_is_not_for_tcgen05(ops):
    """Refused by the kernel's own rule, and taken by the other kernel: pages of four and of 128 keys, a group that is no power of two."""
    for Hq, Hkv, page in ((8, 2, 4), (8, 2, 128), (6, 2, 16)):
        n, hd = 100, 64
        g = torch.Generator(device="cuda").manual_seed(page)
        q, kp, vp = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((n, Hq, hd), (n // page + 1, Hkv, page, hd), (n // page + 1, Hkv, page, hd)))
        i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
        out = torch.zeros(n, Hq * hd, dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(q, kp, vp, torch.arange(n // page + 1, dtype=torch.int32, device="cuda")[None], i32(0, n), i32(n),
                            torch.zeros(n, dtype=torch.int32, device="cuda"), out, hd ** -0.5, 0, page, 1, n, n, softcap=20.0)
        assert ops.tc._capped[hd, hd].gb_capped_attention_tc_takes(*(t.data_ptr() for t in (q, kp, vp, out)), 1, Hq, Hkv, hd ** -0.5, page, len(kp)) == 0
        flat = lambda t: t.transpose(1, 2).reshape(-1, Hkv, hd)[:n].double().repeat_interleave(Hq // Hkv, 1)
        s = 20.0 * torch.tanh(torch.einsum("ihd,jhd->hij", q.double(), flat(kp)) * hd ** -0.5 / 20.0)
        p = torch.softmax(s.masked_fill(~torch.ones(n, n, dtype=torch.bool, device="cuda").tril(), -float("inf")), -1)
        close(out.view(n, Hq, hd), torch.einsum("hij,jhd->ihd", p, flat(vp)).cpu(), torch.bfloat16, "capped attention")

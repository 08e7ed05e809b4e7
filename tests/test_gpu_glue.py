"""Per-token glue kernels against plain torch fp32 references of the same operations (tolerance 1e-3 of the largest
output unless the output itself is a bf16 tensor, where one bf16 rounding, 2^-8, is allowed)."""

import pytest
import torch
import torch.nn.functional as F

from glue_refs import gdn_ref, rope_ref

pytestmark = pytest.mark.gpu

BF16_ULP = 2.0 ** -8


def close(got, ref, tol):
    err = float((got.float() - ref.float()).abs().max() / ref.float().abs().max().clamp_min(1e-20))
    assert err <= tol, err


@pytest.mark.parametrize("rows,hidden", [(1, 5120), (1, 2048), (3, 640), (8, 5120)])
def test_add_rmsnorm(rows, hidden):
    from ixrun_b200.glue import add_rmsnorm

    h = torch.randn(rows, hidden, device="cuda").bfloat16()
    d = torch.randn(rows, hidden, device="cuda").bfloat16()
    w = (1 + 0.1 * torch.randn(hidden, device="cuda")).bfloat16()
    for delta in (d, None):
        h0 = h.clone()
        hr = (h0 + delta) if delta is not None else h0             # bf16 add, as the eager residual
        v = hr.float()
        ref = (v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-5)).to(torch.bfloat16) * w
        hh = h.clone()
        xn = add_rmsnorm(hh, delta, w, 1e-5)
        assert torch.equal(hh, hr)
        close(xn, ref, BF16_ULP)


def test_swiglu():
    from ixrun_b200.glue import swiglu

    g = torch.randn(17408, device="cuda").bfloat16() * 3
    u = torch.randn(17408, device="cuda").bfloat16()
    close(swiglu(g, u), F.silu(g) * u, BF16_ULP)


@pytest.mark.parametrize("hq,hkv,d,rot,norm", [(16, 8, 128, 128, False), (24, 4, 256, 64, True), (3, 1, 256, 256, False)])
def test_rope_kv_and_attention(hq, hkv, d, rot, norm):
    from ixrun_b200.glue import AttnDecode, rope_kv, rope_tables

    dev, max_seq, ctx = "cuda", 512, 300
    cos, sin = rope_tables(max_seq, rot, 10000.0, dev)
    kc = torch.randn(max_seq, hkv, d, device=dev).bfloat16()
    vc = torch.randn(max_seq, hkv, d, device=dev).bfloat16()
    kc0, vc0 = kc.clone(), vc.clone()
    qg = torch.randn(1, 2 * hq * d, device=dev).bfloat16()          # [q | gate], as a gated attention's projection
    k = torch.randn(1, hkv * d, device=dev).bfloat16()
    v = torch.randn(1, hkv * d, device=dev).bfloat16()
    qn = (1 + 0.1 * torch.randn(d, device=dev)).bfloat16() if norm else None
    kn = (1 + 0.1 * torch.randn(d, device=dev)).bfloat16() if norm else None
    pos = torch.tensor([ctx], dtype=torch.int32, device=dev)

    def hnorm(x, w):
        if w is None:
            return x.float()
        f = x.float()
        return ((f * torch.rsqrt(f.pow(2).mean(-1, keepdim=True) + 1e-6)).to(torch.bfloat16) * w).float()

    q_ref = rope_ref(hnorm(qg[:, :hq * d].view(1, hq, d), qn), cos, sin, pos.long(), rot).to(torch.bfloat16)
    k_ref = rope_ref(hnorm(k.view(1, hkv, d), kn), cos, sin, pos.long(), rot).to(torch.bfloat16)
    q = qg.clone()
    rope_kv(q, k, v, pos, kc, vc, cos, sin, hq, hkv, d, rot_dim=rot, q_norm=qn, k_norm=kn, q_stride=2 * hq * d)
    close(q[:, :hq * d].view(1, hq, d), q_ref, BF16_ULP)
    assert torch.equal(q[:, hq * d:], qg[:, hq * d:])               # the gate half is untouched
    close(kc[ctx], k_ref[0], BF16_ULP)
    assert torch.equal(vc[ctx], v.view(hkv, d))
    mask = torch.ones(max_seq, dtype=torch.bool, device=dev)
    mask[ctx] = False
    assert torch.equal(kc[mask], kc0[mask]) and torch.equal(vc[mask], vc0[mask])

    # attention of the rotated query over positions 0 .. ctx, with and without the sigmoid gate
    rep = hq // hkv
    qq = q[:, :hq * d].view(hq, 1, d).float()
    kk = kc[: ctx + 1].float().repeat_interleave(rep, dim=1).transpose(0, 1)      # [hq, S, d]
    vv = vc[: ctx + 1].float().repeat_interleave(rep, dim=1).transpose(0, 1)
    att = torch.softmax(qq @ kk.transpose(1, 2) * d ** -0.5, dim=-1) @ vv         # [hq, 1, d]
    ref = att.view(hq * d)
    for splits in (1, 7, None):
        ad = AttnDecode(hq, hkv, d, dev, splits=splits)
        out = ad(q[0, :hq * d].contiguous(), kc, vc, pos)
        close(out, ref, BF16_ULP)
    gate = q[0, hq * d:].contiguous()
    out = AttnDecode(hq, hkv, d, dev)(q[0, :hq * d].contiguous(), kc, vc, pos, gate=gate)
    close(out, (ref.to(torch.bfloat16) * torch.sigmoid(gate.float()).to(torch.bfloat16)).float(), 2 * BF16_ULP)
    # a context of one position
    p0 = torch.zeros(1, dtype=torch.int32, device=dev)
    out = AttnDecode(hq, hkv, d, dev)(q[0, :hq * d].contiguous(), kc, vc, p0)
    close(out, vc[0].float().repeat_interleave(rep, dim=0).reshape(-1), BF16_ULP)


@pytest.mark.parametrize("ctx", [1, 63, 64, 65, 193, 700])
@pytest.mark.parametrize("hq,hkv,d,splits", [(4, 2, 64, 3), (16, 8, 128, 18), (6, 2, 256, 5), (5, 1, 128, 1), (8, 1, 64, 256),
                                             (4, 4, 64, 5), (5, 1, 64, 1), (14, 2, 64, 18)])
def test_attn_decode_parts(hq, hkv, d, splits, ctx):
    """Chunks of 64 positions: one position, one short of a chunk, a whole one, one more, more chunks than parts; one part
    and the most.  What lies in the cache beyond the position (NaN here) is read ahead and must not count; a sequence gets
    the same bits alone (many CTAs) and among 24 (few, which take several parts each); the two-launch form of the C
    interface agrees to the rounding of its joining sums (bf16 outputs: one unit in the last place, 2^-7 of a value)."""
    from ixrun_b200 import _lib
    from ixrun_b200.glue import AttnDecode

    dev, max_seq, b = "cuda", 760, 24
    gen = torch.Generator(device=dev).manual_seed(ctx)
    kc = torch.randn(b, max_seq, hkv, d, generator=gen, device=dev).bfloat16()
    vc = torch.randn(b, max_seq, hkv, d, generator=gen, device=dev).bfloat16()
    q = torch.randn(b, hq * d, generator=gen, device=dev).bfloat16()
    gate = torch.randn(b, hq * d, generator=gen, device=dev).bfloat16()
    pos = (torch.arange(b, device=dev, dtype=torch.int32) * 13 + ctx - 1).clamp_(max=max_seq - 1)
    for r in range(b):
        kc[r, int(pos[r]) + 1:] = float("nan")
        vc[r, int(pos[r]) + 1:] = float("nan")
    many = AttnDecode(hq, hkv, d, dev, splits=splits, batch=b)
    out = many(q, kc, vc, pos, gate=gate, gate_row_stride=hq * d)
    assert not bool(many.tickets.any())
    one = AttnDecode(hq, hkv, d, dev, splits=splits)
    for r in (0, 1, 7, 23):
        alone = one(q[r], kc[r], vc[r], pos[r:r + 1], gate=gate[r])
        assert torch.equal(alone, out[r])
        n = int(pos[r]) + 1
        s = torch.einsum("ghd,sgd->ghs", q[r].double().view(hkv, hq // hkv, d), kc[r, :n].double()) * d ** -0.5
        ref = torch.einsum("ghs,sgd->ghd", s.softmax(-1), vc[r, :n].double()).reshape(-1)
        ref = ref.bfloat16() * torch.sigmoid(gate[r].float()).bfloat16()
        close(alone, ref, 2 * BF16_ULP)
        two = torch.empty_like(alone)
        _lib.check(_lib.lib().ixb_attn_decode(q[r].data_ptr(), kc[r].data_ptr(), vc[r].data_ptr(), pos[r:].data_ptr(),
                                              gate[r].data_ptr(), d, two.data_ptr(), one.scratch.data_ptr(), one.scratch.numel(),
                                              hq, hkv, d, splits, d ** -0.5, 1, 0, 0, 0, _lib.stream_ptr(q.device)))
        assert ((two.float() - alone.float()).abs() <= 2.0 ** -7 * alone.float().abs() + 2.0 ** -16).all()
    assert not bool(one.tickets.any())


@pytest.mark.parametrize("groups", [40, 200, 240, 300])
@pytest.mark.parametrize("hq,hkv,d,splits", [(2, 1, 64, 18), (16, 8, 128, 18), (16, 8, 128, 3), (12, 4, 128, 65), (16, 4, 128, 9),
                                             (12, 2, 64, 18), (3, 3, 128, 1), (6, 2, 256, 9), (8, 2, 256, 2)])
def test_attn_decode_one_cta_per_group(hq, hkv, d, splits, groups):
    """From a few sequences to so many that one CTA takes all parts of a group, through all forms of the kernel: no position
    (NaN), one, the edges of a chunk and of a part, more parts than are kept in shared memory, the whole cache.  Each sequence has
    the bits that it has alone."""
    from ixrun_b200.glue import AttnDecode

    dev, max_seq, b = "cuda", 1300, -(-groups // hkv)
    gen = torch.Generator(device=dev).manual_seed(hq)
    kc = torch.randn(b, max_seq, hkv, d, generator=gen, device=dev).bfloat16()
    vc = torch.randn(b, max_seq, hkv, d, generator=gen, device=dev).bfloat16()
    q = torch.randn(b, hq * d, generator=gen, device=dev).bfloat16()
    gate = torch.randn(b, hq * d, generator=gen, device=dev).bfloat16()
    edges = [-1, 0, 62, 63, 64, 127, 128, 64 * splits - 1, 64 * splits, 64 * splits + 64, 700, max_seq - 1]
    pos = torch.tensor([edges[i % len(edges)] for i in range(b)], dtype=torch.int32, device=dev).clamp_(max=max_seq - 1)
    beyond = torch.arange(max_seq, device=dev)[None, :] > pos[:, None]
    kc[beyond] = float("nan")
    vc[beyond] = float("nan")
    many = AttnDecode(hq, hkv, d, dev, splits=splits, batch=b)
    one = AttnDecode(hq, hkv, d, dev, splits=splits)
    for g in (None, gate):
        out = many(q, kc, vc, pos, gate=g, gate_row_stride=hq * d if g is not None else 0)
        assert not bool(many.tickets.any())
        for r in [*range(min(b, len(edges))), b - 1]:
            alone = one(q[r], kc[r], vc[r], pos[r:r + 1], gate=None if g is None else g[r])
            assert torch.equal(alone.view(torch.int16), out[r].view(torch.int16))


class _NoLaunch:
    """stands in for the C library: a call that gets as far as a launch fails the test instead of handing a host pointer on"""

    def __getattr__(self, name):
        return lambda *a: pytest.fail(f"{name} was called")


@pytest.mark.parametrize("host", ["q", "pos", "gate", "out"])
def test_attn_decode_and_rope_refuse_host_tensors(monkeypatch, host):
    from ixrun_b200 import _lib
    from ixrun_b200.glue import AttnDecode, rope_kv, rope_tables

    bf = dict(dtype=torch.bfloat16, device="cuda")
    t = {"q": torch.zeros(256, **bf), "gate": torch.zeros(256, **bf), "out": torch.zeros(256, **bf),
         "pos": torch.zeros(1, dtype=torch.int32, device="cuda")}
    kc, vc = torch.zeros(32, 2, 64, **bf), torch.zeros(32, 2, 64, **bf)
    kv = torch.zeros(1, 128, **bf)
    cos, sin = rope_tables(32, 64, 10000.0, "cuda")
    ad = AttnDecode(4, 2, 64, "cuda")
    ad(t["q"], kc, vc, t["pos"], out=t["out"], gate=t["gate"])
    t[host] = t[host].cpu()
    monkeypatch.setattr(_lib, "lib", lambda: _NoLaunch())
    with pytest.raises(ValueError):
        ad(t["q"], kc, vc, t["pos"], out=t["out"], gate=t["gate"])
    if host in ("q", "pos"):
        with pytest.raises(ValueError):
            rope_kv(t["q"], kv, kv, t["pos"], kc, vc, cos, sin, 4, 2, 64, q_stride=256)


@pytest.mark.parametrize("view", [lambda c: c.view(96, 128), lambda c: c.view(-1), lambda c: c.view(1, 96, 128), lambda c: c.view(1, 96, 2, 64)])
def test_attn_decode_takes_a_cache_of_any_shape(view):
    """One sequence's cache is max_seq * hkv * head_dim numbers; the same bits in every shape."""
    from ixrun_b200.glue import AttnDecode

    bf = dict(dtype=torch.bfloat16, device="cuda")
    kc, vc, q = torch.randn(96, 2, 64, **bf), torch.randn(96, 2, 64, **bf), torch.randn(256, **bf)
    pos = torch.tensor([80], dtype=torch.int32, device="cuda")
    ad = AttnDecode(4, 2, 64, "cuda", splits=3)
    assert torch.equal(ad(q, view(kc), view(vc), pos), ad(q, kc, vc, pos))


def test_attn_decode_reads_ahead_in_what_both_caches_hold(monkeypatch):
    """The rows that the kernel may touch before it knows the position, as the library is told: those of the shorter cache."""
    from ixrun_b200 import _lib
    from ixrun_b200.glue import AttnDecode

    seen = []

    class Record:
        def ixb_attn_decode_join(self, *a):
            seen.append(a[-2])
            return 0

    bf = dict(dtype=torch.bfloat16, device="cuda")
    pos = torch.zeros(2, dtype=torch.int32, device="cuda")
    one, two = AttnDecode(4, 2, 64, "cuda", splits=3), AttnDecode(4, 2, 64, "cuda", splits=3, batch=2)
    monkeypatch.setattr(_lib, "lib", lambda: Record())
    for k, v, want in ((96, 96, 96), (96, 70, 70), (70, 96, 70)):
        one(torch.zeros(256, **bf), torch.zeros(k, 2, 64, **bf), torch.zeros(v, 2, 64, **bf), pos)
        assert seen.pop() == want
    two(torch.zeros(2, 256, **bf), torch.zeros(3, 96, 2, 64, **bf), torch.zeros(3, 96, 2, 64, **bf), pos)
    assert seen.pop() == 96


def test_attn_decode_recovers_from_overlapping_launches():
    """Launches of one object on two streams at once, with different numbers of parts, spoil each other's results but not
    those of later calls: the tickets are zero again."""
    from ixrun_b200.glue import AttnDecode

    bf = dict(dtype=torch.bfloat16, device="cuda")
    kc, vc, q = torch.randn(1200, 2, 128, **bf), torch.randn(1200, 2, 128, **bf), torch.randn(512, **bf)
    pos = [torch.tensor([n], dtype=torch.int32, device="cuda") for n in (1100, 170, 20, -1)]
    ad = AttnDecode(4, 2, 128, "cuda", splits=18)
    want = [ad(q, kc, vc, p) for p in pos[:3]]
    streams = [torch.cuda.Stream() for _ in pos]
    torch.cuda.synchronize()
    for _ in range(100):
        for s, p in zip(streams, pos):
            with torch.cuda.stream(s):
                ad(q, kc, vc, p)
    torch.cuda.synchronize()
    assert not bool(ad.tickets.any())
    for p, w in zip(pos, want):
        assert torch.equal(ad(q, kc, vc, p), w)


def test_attn_decode_is_ready_for_any_stream():
    """An object made on a busy stream, in memory that held something else, and first called on another stream."""
    from ixrun_b200.glue import AttnDecode

    bf = dict(dtype=torch.bfloat16, device="cuda")
    kc, vc, q = torch.randn(1200, 2, 128, **bf), torch.randn(1200, 2, 128, **bf), torch.randn(512, **bf)
    pos = torch.tensor([1100], dtype=torch.int32, device="cuda")
    want = AttnDecode(4, 2, 128, "cuda", splits=18)(q, kc, vc, pos)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        held = torch.full((4,), 7, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        del held                                                   # its block is the next one of this size on this stream
        torch.cuda._sleep(20_000_000)
        ad = AttnDecode(4, 2, 128, "cuda", splits=18)
    assert torch.equal(ad(q, kc, vc, pos), want)


@pytest.mark.parametrize("rows,pos0", [(1, 0), (1, 90), (63, 0), (64, 64), (65, 0), (200, 37)])
@pytest.mark.parametrize("hq,hkv,d", [(4, 2, 64), (3, 3, 128), (6, 1, 128)])
def test_attn_prefill(hq, hkv, d, rows, pos0):
    """Row and key tiles of 64: one row, one short of a tile, a whole one, one more; from the start and behind a context.
    Bound: the bf16 output is off by at most half a unit in the last place, 2^-8 of the value (8 significant bits; the
    value may sit at the bottom of its binade); the fp32 exponentials and sums add less than 2^-16 of the largest value."""
    from ixrun_b200.glue import attn_prefill

    max_seq, dev = pos0 + rows + 30, "cuda"
    qkv = torch.randn(rows, (hq + 2 * hkv) * d, device=dev).bfloat16()        # q is a column slice of a wider matrix
    kc = torch.randn(max_seq, hkv, d, device=dev).bfloat16()
    vc = torch.randn(max_seq, hkv, d, device=dev).bfloat16()
    out = attn_prefill(qkv[:, :hq * d], kc, vc, pos0, hq, hkv, d)
    n = pos0 + rows
    q = qkv[:, :hq * d].double().view(rows, hkv, hq // hkv, d)
    s = torch.einsum("rghd,sgd->rghs", q, kc[:n].double()) * d ** -0.5
    mask = torch.arange(n, device=dev)[None, :] <= pos0 + torch.arange(rows, device=dev)[:, None]
    p = s.masked_fill(~mask[:, None, None, :], -torch.inf).softmax(-1)
    ref = torch.einsum("rghs,sgd->rghd", p, vc[:n].double()).reshape(rows, hq * d)
    err = (out.double() - ref).abs()
    assert (err <= ref.abs() * BF16_ULP + 2.0 ** -16 * vc.abs().max()).all(), float(err.max())


def test_conv_update():
    from ixrun_b200.glue import conv_update

    c, k = 10240, 4
    w = torch.randn(c, k, device="cuda").bfloat16()
    bias = torch.randn(c, device="cuda").bfloat16()
    state = torch.randn(c, k - 1, device="cuda").bfloat16()
    hist = state.clone()
    for step in range(5):
        x = torch.randn(c, device="cuda").bfloat16()
        full = torch.cat([hist.float(), x.float()[:, None]], dim=1)                 # [C, K]
        ref = F.silu((full * w.float()).sum(-1) + bias.float())
        y = conv_update(x, state, w, bias if step % 2 == 0 else None)
        if step % 2:
            ref = F.silu((full * w.float()).sum(-1))
        close(y, ref, BF16_ULP)
        hist = full[:, 1:].to(torch.bfloat16)
        assert torch.equal(state, hist)


@pytest.mark.parametrize("hk,hv", [(16, 48), (2, 6), (1, 1)])
def test_gdn_step(hk, hv):
    from ixrun_b200.glue import gdn_step

    dev = "cuda"
    S = torch.randn(hv, 128, 128, device=dev) * 0.1
    A_log = torch.randn(hv, device=dev) * 0.5
    dt_bias = torch.randn(hv, device=dev) * 0.5
    norm_w = (1 + 0.1 * torch.randn(128, device=dev)).bfloat16()
    S_gpu = S.clone()
    for step in range(3):
        qkv = torch.randn(2 * hk * 128 + hv * 128, device=dev).bfloat16()
        z = torch.randn(hv * 128, device=dev).bfloat16()
        a = torch.randn(hv, device=dev).bfloat16()
        b = torch.randn(hv, device=dev).bfloat16()
        ref, S = gdn_ref(qkv, z, a, b, A_log, dt_bias, norm_w, S, hk, hv, 1e-6)
        out = gdn_step(qkv, z, a, b, A_log, dt_bias, norm_w, S_gpu, hk, hv, 1e-6)
        close(S_gpu, S, 1e-4)
        close(out, ref, 2 * BF16_ULP)


@pytest.mark.parametrize("hk,hv", [(16, 48), (2, 6), (1, 1)])
def test_gdn_conv_step_equals_conv_then_gdn(hk, hv):
    """The fused kernel (conv history kept twice, read copy pos & 1, write the other) gives the bits of the conv
    kernel followed by the recurrent kernel, step after step."""
    from ixrun_b200.glue import conv_update, gdn_conv_step, gdn_step

    dev = "cuda"
    C = (2 * hk + hv) * 128
    conv_w = (torch.randn(C, 4, device=dev) * 0.3).bfloat16()
    A_log = torch.randn(hv, device=dev) * 0.5
    dt_bias = torch.randn(hv, device=dev) * 0.5
    norm_w = (1 + 0.1 * torch.randn(128, device=dev)).bfloat16()
    S_a = torch.randn(hv, 128, 128, device=dev) * 0.1
    S_b = S_a.clone()
    hist = torch.randn(C, 3, device=dev).bfloat16()
    start = 5                                              # an odd first position: the first step reads copy 1
    state2 = torch.zeros(2, C, 3, dtype=torch.bfloat16, device=dev)
    state2[start & 1] = hist
    pos = torch.tensor([start], dtype=torch.int32, device=dev)
    for step in range(4):
        qkv = torch.randn(C, device=dev).bfloat16()
        z = torch.randn(hv * 128, device=dev).bfloat16()
        a = torch.randn(hv, device=dev).bfloat16()
        b = torch.randn(hv, device=dev).bfloat16()
        ref = gdn_step(conv_update(qkv, hist, conv_w), z, a, b, A_log, dt_bias, norm_w, S_a, hk, hv, 1e-6)
        out = gdn_conv_step(qkv, state2, conv_w, pos, z, a, b, A_log, dt_bias, norm_w, S_b, hk, hv, 1e-6)
        assert torch.equal(out, ref) and torch.equal(S_a, S_b)
        pos += 1
        assert torch.equal(state2[int(pos.item()) & 1], hist)
